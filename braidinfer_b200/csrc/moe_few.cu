// The experts' products of steps of few tokens:  out[slot, m] = sum_k x[row or slot, k] * w[expert of the slot, m, k], bfloat16, float32 sums,
// for slots sorted by expert (moe.cu, moe_plan with tiles of 32 slots; an expert has one tile, whose slots are at most the step's 8 tokens).
//
// Bound by the weights' bytes.  On pairs of SMs (moe_tc.cu) a tile of 256 weight rows walks its k blocks one round trip of six stages at a
// time, 0.36 us each, on as many pairs as there are tiles: a few experts leave pairs idle and the second product's long k is a chain.  Here
// a unit is 16 weight rows of one expert (8 rows of gate and the 8 of up that go with them), as in gemm_few.cu: four warps share k, the
// weights go straight to the operand registers, and their sums meet in shared memory.  The CTAs that
// fit (four an SM) walk the units and ask for the next one's weights before they finish one; with 740 CTAs, of which 148 wait for a place,
// 197.7 us read 240.7, with a CTA a unit 203.8.  The tokens' rows are read where they lie: no copy of them.
// Both products of a step, us, against the copy of the rows and pairs of SMs (floor: the chosen experts' bytes at 6.4 TB/s):
//   64 experts of 1408 x 2048, 6 a token:   1 token 32 / 44 (16), 4 tokens 73 / 91 (54), 8 tokens 116 / 134 (95)
//   8 experts of 7168 x 4096, 2 a token:    1 token 79 / 106 (55), 4 tokens 171 / 206 (138), 8 tokens 229 / 253 (193)
//   16 experts of 1024 x 1024, 2 a token:   1 token 13 / 28 (2), 8 tokens 26 / 40 (10)
// Two blocks of 8 slots (9 to 16 tokens) hold too many registers: 206 / 155 at 12 tokens of the first, so steps above 8 stay on the pairs.
#include "few.cuh"

#define MF_WARPS 4
#define MF_TURNS 4                 // turns of 64 numbers of k in flight a warp
#define MF_CHUNK 32                // slots of a plan tile
#define MF_TOKENS 8                // of them in use at most
#define MF_CTAS 4                  // on an SM: 16 warps with 8 KB of weights each on their way

struct MoeFewArgs {
    const __nv_bfloat16 *x, *w;
    __nv_bfloat16* out;
    const int *tile_expert, *meta, *slot_pair;
    const float* in_wgt;           // gated: a weight a pair on the expert's input, or null
    long long ldx, ldo;
    int k8, w_rows, m_out, units, max_tiles, top;      // units: of an expert; top: choices a token, 0: x's rows are the slots'
};

// MODE 0 product, 1 silu(gate) * up over rows interleaved in blocks of 16, 2 relu(product)^2.
template <int MODE>
__global__ void __launch_bounds__(MF_WARPS * 32, MF_CTAS)
moe_few_kernel(const __grid_constant__ MoeFewArgs a) {
    constexpr int W = MF_WARPS, U = MF_TURNS, OUTS = MODE == 1 ? 8 : 16;
    __shared__ float part[W][MF_TOKENS][17];                 // [warp][slot][tile row]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    pdl_wait();
    const int n_units = min(a.meta[0], a.max_tiles) * a.units, turns = (a.k8 + 7) / 8;
    const uint4* wr[2];
    const uint4* xr;
    uint4 wv[U][2][2];
    int tile = 0, m = 0;
    auto fetch = [&](int u, int turn) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = turn * 8 + h * 4 + q;
#pragma unroll
            for (int r = 0; r < 2; ++r) wv[u][r][h] = c < a.k8 ? few_load_weights(wr[r] + c) : zero;
        }
    };
    auto start = [&](int unit) {                             // its weights on their way, its slots' rows
        tile = unit / a.units;
        m = unit - tile * a.units;
        const size_t row0 = (size_t)a.tile_expert[tile] * a.w_rows;
        int r0, r1;
        if (MODE == 1) {
            r0 = (m >> 1) * 32 + (m & 1) * 8 + g;            // every block of 32 rows is stored whole
            r1 = r0 + 16;
        } else {
            r0 = min(m * 16 + g, a.m_out - 1);
            r1 = min(m * 16 + g + 8, a.m_out - 1);
        }
        wr[0] = reinterpret_cast<const uint4*>(a.w + (row0 + r0) * a.k8 * 8);
        wr[1] = reinterpret_cast<const uint4*>(a.w + (row0 + r1) * a.k8 * 8);
#pragma unroll
        for (int u = 0; u < U; ++u) fetch(u, warp + u * W);
        const int slot = tile * MF_CHUNK + g, pair = a.slot_pair[slot];
        xr = pair < 0 ? nullptr : reinterpret_cast<const uint4*>(a.x + (size_t)(a.top ? pair / a.top : slot) * a.ldx);
    };
    int unit = blockIdx.x;
    if (unit < n_units) start(unit);
    while (unit < n_units) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int t0 = warp; t0 < turns; t0 += U * W) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int turn = t0 + u * W;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = turn * 8 + h * 4 + q;
                    const uint4 xv = (xr && c < a.k8) ? xr[c] : zero;
                    few_mma(acc, wv[u][0][h].x, wv[u][1][h].x, wv[u][0][h].y, wv[u][1][h].y, xv.x, xv.y);
                    few_mma(acc, wv[u][0][h].z, wv[u][1][h].z, wv[u][0][h].w, wv[u][1][h].w, xv.z, xv.w);
                }
                if (turn + U * W < turns) fetch(u, turn + U * W);
            }
        }
        const int tile_now = tile, m_now = m;
        unit += gridDim.x;
        if (unit < n_units) start(unit);
        part[warp][2 * q][g] = acc[0];
        part[warp][2 * q + 1][g] = acc[1];
        part[warp][2 * q][g + 8] = acc[2];
        part[warp][2 * q + 1][g + 8] = acc[3];
        __syncthreads();
        for (int i = threadIdx.x; i < MF_TOKENS * OUTS; i += W * 32) {
            const int o = i % OUTS, n = i / OUTS, at = m_now * OUTS + o, slot = tile_now * MF_CHUNK + n;
            const int pair = a.slot_pair[slot];
            if (at >= a.m_out || pair < 0) continue;
            float v = 0.f, up = 0.f;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                v += part[w][n][o];
                if (MODE == 1) up += part[w][n][o + 8];
            }
            if (MODE == 1) {
                const float s = a.in_wgt ? a.in_wgt[pair] : 1.f;
                v = silu_to_bf16(v * s) * (up * s);
            }
            if (MODE == 2) v = v > 0.f ? v * v : v < 0.f ? 0.f : v * 0.f;        // (a NaN stays one)
            a.out[(size_t)slot * a.ldo + at] = __float2bfloat16_rn(v);
        }
        __syncthreads();
    }
    pdl_trigger();                                           // (see gemm_few.cu)
}

template <int MODE>
static int launch_moe_few(const MoeFewArgs& a, cudaStream_t s) {
    const long long units = (long long)a.max_tiles * a.units;
    const dim3 grid((unsigned)(units < 148 * MF_CTAS ? units : 148 * MF_CTAS));
    braid_launch(moe_few_kernel<MODE>, grid, dim3(MF_WARPS * 32), 0, s, a);
    BRAID_LAUNCH_CHECK();
}

// Steps of `rows` <= 8 tokens, each of which chose different experts.  w: experts x w_rows rows of k (mode 1: gate and up interleaved in
// blocks of 16 rows); x: the step's rows (top > 0: choices a token) or the slots'.
extern "C" int braid_moe_few(const void* x, long long ldx, const void* w, void* out, long long ldo, const int* slot_pair, const int* tile_expert,
                             const int* meta, int mode, int rows, int top, int w_rows, int m_out, int k, int max_tiles, const float* in_wgt, void* stream) {
    if (max_tiles <= 0 || m_out <= 0 || rows <= 0) return BRAID_OK;
    if (mode < 0 || mode > 2) BRAID_REFUSE("moe_few: unknown mode %d", mode);
    if (rows > MF_TOKENS) BRAID_REFUSE("moe_few: %d rows (at most %d)", rows, MF_TOKENS);
    if (k <= 0 || k % 8 || ldx % 8 || ldo < m_out || (((uintptr_t)x | (uintptr_t)w) & 15)) BRAID_REFUSE("moe_few: k=%d must be a multiple of 8, rows must start on 16 bytes", k);
    if (w_rows != (mode == 1 ? 2 * ((m_out + 15) / 16 * 16) : m_out)) BRAID_REFUSE("moe_few: %d weight rows an expert do not fit %d outputs", w_rows, m_out);
    if (in_wgt && mode != 1) BRAID_REFUSE("moe_few: a weight on the expert's input goes with the gated first product");
    const MoeFewArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)out, tile_expert, meta, slot_pair, in_wgt, ldx, ldo, k / 8, w_rows,
                       m_out, mode == 1 ? (m_out + 7) / 8 : (m_out + 15) / 16, max_tiles, top};
    cudaStream_t s = (cudaStream_t)stream;
    return mode == 0 ? launch_moe_few<0>(a, s) : mode == 1 ? launch_moe_few<1>(a, s) : launch_moe_few<2>(a, s);
}
