// bfloat16 matrix product of a few tokens, in one kernel:
//   out[n, m] = sum_k x[n, k] * w[m, k],   n <= 16, float32 accumulation.
//
// Bound by the weights' bytes, and for the smaller matrices by latency.  The stream-k form of gemm_tc.cu spreads any shape evenly
// over the SMs, but its partial sums need a second kernel: 5 to 7 us for the two where the weights' bytes take 0.3 to 3.5.
// Here a CTA owns 16 weight rows and all of k, so the sum is finished where it is made.  The W warps of the CTA share k, 64
// numbers a turn each, and stream the weights straight from memory into the operand registers of mma.sync m16n8k16: which 16
// numbers of k one MMA takes is free as long as both operands agree, so a lane's 16 bytes of a row are the k pairs of two MMAs and
// nothing passes through shared memory (the tensor cores are idle most of the time either way; tcgen05 would put TMA, two
// barriers and tensor memory between a weight and its product).  U turns are in flight a warp, the first of them asked for before the
// dependency wait: no kernel writes weights.  The warps' sums meet in shared memory in the order of the warps.
//
// Epilogues: 0 store, 1 float32 residual sum, 2 gated unit, 3 act(product) times a number of the row's token from a table.  A gated tile is 8 gate rows and the 8 up rows that go with
// them (rows interleaved in blocks of 16, see gemm_tc.cu), so that both halves meet in one CTA.  A row scale that x still
// wants (rowscale.cuh) multiplies the finished sums of 0 and 2.
//
// Measured in graphs of back-to-back products on weights that do not fit L2, us, beside stream-k and its reduce kernel (in brackets what
// the bytes take at 6.55 TB/s), 8 tokens: 1024 x 1024 2.8 beside 5.7 (0.3), 1024 x 2816 3.7 / 6.9 (0.9), 2048 x 2048 3.9 / 6.4
// (1.3), 2048 x 5632 7.7 / 10.1 (3.5), 3072 x 2048 4.8 / 7.0 (1.9), 11264 x 2048 10.2 / 11.4 (7.0), 28672 x 4096 43.4 / 40.8
// (35.9): tokens come through L1 once a CTA, which costs most where the CTAs are many.  Between the other kernels of a decode step the
// larger products lose that lead, because their CTAs come to lie on the SMs that the kernel before leaves first (32 layers with
// 4096 x 4096 and 4096 x 14336 so: 64.5 beside 51.6 ms a turn of one sequence): `few_rows_pay` (parts/linear.py) draws the line.
#include "common.cuh"
#include "rowscale.cuh"
#include "few.cuh"

#define FEW_MAX_ROWS 16

struct GemmFewArgs {
    const void* x;              // bfloat16, or float32 that is rounded as it is read (XF)
    const __nv_bfloat16* w;
    void* out;                  // mode 0: bf16/f32; 1: f32; 2: bf16/f32
    const float* res;           // mode 1 (may be out)
    int n_rows, m_out, k8;      // m_out: outputs; k8: k / 8
    long long ldx, ldw, ldo;
    int out_f32, act;
    RowScaleArgs scale;
    const __nv_bfloat16* table; // mode 3: [vocab, table_stride], output o of row n times table[ids[n], o]
    long long table_stride;
    const int* ids;
    int vocab;
};

// eight numbers of a row, in bfloat16
template <bool XF>
__device__ __forceinline__ uint4 few_load_x(const void* x, size_t at) {
    if (!XF) return *reinterpret_cast<const uint4*>((const __nv_bfloat16*)x + at);
    const float4 a = *reinterpret_cast<const float4*>((const float*)x + at), b = *reinterpret_cast<const float4*>((const float*)x + at + 4);
    const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w), __floats2bfloat162_rn(b.x, b.y), __floats2bfloat162_rn(b.z, b.w)};
    return *reinterpret_cast<const uint4*>(p);
}

// NT: blocks of 8 tokens.
template <int MODE, int NT, int W, int U, bool XF = false>
__global__ void __launch_bounds__(W * 32)
gemm_few_bf16_kernel(GemmFewArgs a) {
    __shared__ float part[W][NT][8][17];                     // [warp][token block][token][tile row]
    __shared__ float rs[FEW_MAX_ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int tile = blockIdx.x;
    // the weight rows of tile rows g and g + 8
    int r0, r1;
    if (MODE == 2) {
        r0 = (tile >> 1) * 32 + (tile & 1) * 8 + g;          // every block of 32 rows is stored whole
        r1 = r0 + 16;
    } else {
        r0 = min(tile * 16 + g, a.m_out - 1);
        r1 = min(tile * 16 + g + 8, a.m_out - 1);
    }
    const uint4* wr[2] = {reinterpret_cast<const uint4*>(a.w + (size_t)r0 * a.ldw), reinterpret_cast<const uint4*>(a.w + (size_t)r1 * a.ldw)};
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 wv[U][2][2];
    auto fetch = [&](int u, int turn) {                      // turn: 64 numbers of k, a lane takes 8 of either half
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = turn * 8 + h * 4 + q;
#pragma unroll
            for (int r = 0; r < 2; ++r) wv[u][r][h] = c < a.k8 ? few_load_weights(wr[r] + c) : zero;
        }
    };
#pragma unroll
    for (int u = 0; u < U; ++u) fetch(u, warp + u * W);
    pdl_wait();
    if (a.scale.shares && warp == W - 1 && lane < a.n_rows) rs[lane] = row_scale_of(a.scale, lane);
    size_t xr[NT];
    bool live[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        live[n] = n * 8 + g < a.n_rows;
        xr[n] = (size_t)(live[n] ? n * 8 + g : 0) * a.ldx;
    }
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    const int turns = (a.k8 + 7) / 8;
    for (int t0 = warp; t0 < turns; t0 += U * W) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int turn = t0 + u * W;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = turn * 8 + h * 4 + q;
                    const uint4 xv = (live[n] && c < a.k8) ? few_load_x<XF>(a.x, xr[n] + c * 8) : zero;
                    few_mma(acc[n], wv[u][0][h].x, wv[u][1][h].x, wv[u][0][h].y, wv[u][1][h].y, xv.x, xv.y);
                    few_mma(acc[n], wv[u][0][h].z, wv[u][1][h].z, wv[u][0][h].w, wv[u][1][h].w, xv.z, xv.w);
                }
            fetch(u, turn + U * W);
        }
    }
    // only here: a successor whose CTAs take their places while this kernel's are still spread unevenly over the SMs keeps those places
    // (a turn of 8 sequences of a four-layer model of width 1024: 7.3 ms with the release at the top, 6.7 here)
    pdl_trigger();
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        part[warp][n][2 * q][g] = acc[n][0];
        part[warp][n][2 * q + 1][g] = acc[n][1];
        part[warp][n][2 * q][g + 8] = acc[n][2];
        part[warp][n][2 * q + 1][g + 8] = acc[n][3];
    }
    __syncthreads();
    constexpr int OUTS = MODE == 2 ? 8 : 16;                 // outputs of a tile
    for (int i = threadIdx.x; i < NT * 8 * OUTS; i += W * 32) {
        const int o = i % OUTS, n = i / OUTS, m = tile * OUTS + o;
        if (m >= a.m_out || n >= a.n_rows) continue;
        float v = 0.f, up = 0.f;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            v += part[w][n >> 3][n & 7][o];
            if (MODE == 2) up += part[w][n >> 3][n & 7][o + 8];
        }
        const size_t at = (size_t)n * a.ldo + m;
        if (MODE == 1) {
            ((float*)a.out)[at] = a.res[at] + v;
            continue;
        }
        if (MODE == 3) {
            const int id = min(max(a.ids[n], 0), a.vocab - 1);
            ((__nv_bfloat16*)a.out)[at] = __float2bfloat16_rn(glu_act(v, a.act) * __bfloat162float(a.table[(size_t)id * a.table_stride + m]));
            continue;
        }
        const float s = a.scale.shares ? rs[n] : 1.f;
        v *= s;
        if (MODE == 2) v = glu_act_fast(v, a.act) * (up * s);
        if (a.out_f32) ((float*)a.out)[at] = v;
        else ((__nv_bfloat16*)a.out)[at] = __float2bfloat16_rn(v);
    }
}

template <int MODE, int NT>
static void launch_few_bf16(const GemmFewArgs& a, int tiles, cudaStream_t s) {
    // As many warps a CTA as give the machine some 2,500 and more, each with two turns of 64 numbers at least; a CTA an SM keeps
    // four turns a warp in flight, where more share an SM two do (8 tokens, us with 16 warps and 2 / 4 turns: 4096 x 4096 8.9 /
    // 10.6, 2048 x 2048 4.4 / 3.9).
    const int turns = (a.k8 + 7) / 8;
    const dim3 grid(tiles);
    if (tiles <= 256 && turns >= 32) {
        if (tiles <= 148) braid_launch(gemm_few_bf16_kernel<MODE, NT, 16, 4>, grid, dim3(512), 0, s, a);
        else braid_launch(gemm_few_bf16_kernel<MODE, NT, 16, 2>, grid, dim3(512), 0, s, a);
    } else if (tiles > 148 && tiles <= 450) {
        braid_launch(gemm_few_bf16_kernel<MODE, NT, 8, 2>, grid, dim3(256), 0, s, a);
    } else {
        braid_launch(gemm_few_bf16_kernel<MODE, NT, 4, 4>, grid, dim3(128), 0, s, a);
    }
}

// mode 0 store, 1 residual sum (float32), 2 gated unit over interleaved gate/up rows, its activation in bits 4..7.
extern "C" int braid_gemm_few(const void* x, const void* w, void* out, const float* res, int out_dtype, int mode, int n_rows, int m_out,
                              int k_in, long long ldx, long long ldw, long long ldo, const float* shares, int n_shares,
                              long long share_stride, float width, float eps, void* stream) {
    if (n_rows <= 0 || m_out <= 0) return BRAID_OK;
    const int act = (mode >> 4) & 15;
    mode &= 15;
    if (mode < 0 || mode > 2) BRAID_REFUSE("gemm_few: unknown epilogue %d", mode);
    if (act >= BRAID_ACT_COUNT || (act && mode != 2)) BRAID_REFUSE("gemm_few: unknown activation %d for epilogue %d", act, mode);
    if (n_rows > FEW_MAX_ROWS) BRAID_REFUSE("gemm_few: %d rows (at most %d)", n_rows, FEW_MAX_ROWS);
    if (k_in <= 0 || k_in % 8 || ldx % 8 || ldw % 8) BRAID_REFUSE("gemm_few: k=%d and the row strides (%lld, %lld) must be multiples of 8", k_in, ldx, ldw);
    if (((uintptr_t)x | (uintptr_t)w) & 15) BRAID_REFUSE("gemm_few: operands must start on 16 bytes");
    if (mode == 1 && (!res || out_dtype != BRAID_F32)) BRAID_REFUSE("gemm_few: the residual epilogue writes float32 and needs res");
    if (out_dtype != BRAID_F32 && out_dtype != BRAID_BF16) BRAID_REFUSE("gemm_few: unknown out dtype code %d", out_dtype);
    const RowScaleArgs rsa{shares, n_shares, share_stride, width, eps};
    if (const char* p = row_scale_problem(rsa, n_rows)) BRAID_REFUSE("gemm_few: row scale: %s", p);
    if (shares && mode == 1) BRAID_REFUSE("gemm_few: the residual sum applies no row scale");
    GemmFewArgs a{x, (const __nv_bfloat16*)w, out, res, n_rows, m_out, k_in / 8, ldx, ldw, ldo, out_dtype == BRAID_F32, act, rsa, nullptr, 0, nullptr, 0};
    const int tiles = mode == 2 ? (m_out + 7) / 8 : (m_out + 15) / 16;
    cudaStream_t s = (cudaStream_t)stream;
    if (n_rows <= 8) {
        if (mode == 0) launch_few_bf16<0, 1>(a, tiles, s);
        else if (mode == 1) launch_few_bf16<1, 1>(a, tiles, s);
        else launch_few_bf16<2, 1>(a, tiles, s);
    } else {
        if (mode == 0) launch_few_bf16<0, 2>(a, tiles, s);
        else if (mode == 1) launch_few_bf16<1, 2>(a, tiles, s);
        else launch_few_bf16<2, 2>(a, tiles, s);
    }
    BRAID_LAUNCH_CHECK();
}

// x float32, rounded to bfloat16 as it is read: out[n, o] = act((x w^T)[n, o]) * table[ids[n], col0 + o] in bfloat16 (three kernels of 1.1, 2.0 and
// 1.6 us between the others of a decode step of 8 rows, 128 x 1024: 3.2 in one).
extern "C" int braid_gemm_few_table(const float* x, const void* w, void* out, int n_rows, int m_out, int k_in, long long ldx, long long ldw,
                                    long long ldo, const void* table, long long table_stride, const int* ids, int vocab, int col0, int act,
                                    void* stream) {
    if (n_rows <= 0 || m_out <= 0) return BRAID_OK;
    if (n_rows > FEW_MAX_ROWS) BRAID_REFUSE("gemm_few_table: %d rows (at most %d)", n_rows, FEW_MAX_ROWS);
    if (k_in <= 0 || k_in % 8 || ldx % 4 || ldw % 8 || (((uintptr_t)x | (uintptr_t)w) & 15)) BRAID_REFUSE("gemm_few_table: k=%d must be a multiple of 8 and rows start on 16 bytes", k_in);
    if (act < 0 || act >= BRAID_ACT_COUNT) BRAID_REFUSE("gemm_few_table: unknown activation %d", act);
    if (!table || !ids || vocab <= 0 || col0 < 0) BRAID_REFUSE("gemm_few_table: vocab=%d, col0=%d", vocab, col0);
    const GemmFewArgs a{x, (const __nv_bfloat16*)w, out, nullptr, n_rows, m_out, k_in / 8, ldx, ldw, ldo, 0, act, RowScaleArgs{},
                        (const __nv_bfloat16*)table + col0, table_stride, ids, vocab};
    const dim3 grid((m_out + 15) / 16);
    cudaStream_t s = (cudaStream_t)stream;
    // few CTAs: sixteen warps each, as k allows
    if (n_rows <= 8) {
        if (k_in >= 1024) braid_launch(gemm_few_bf16_kernel<3, 1, 16, 2, true>, grid, dim3(512), 0, s, a);
        else braid_launch(gemm_few_bf16_kernel<3, 1, 4, 4, true>, grid, dim3(128), 0, s, a);
    } else {
        if (k_in >= 1024) braid_launch(gemm_few_bf16_kernel<3, 2, 16, 2, true>, grid, dim3(512), 0, s, a);
        else braid_launch(gemm_few_bf16_kernel<3, 2, 4, 4, true>, grid, dim3(128), 0, s, a);
    }
    BRAID_LAUNCH_CHECK();
}
