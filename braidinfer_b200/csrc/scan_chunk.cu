// The linear recurrence of scan.cu over chunks of a prompt, for bfloat16 rows, with a decay a key channel (gated linear attention) or
// one constant decay a head (lightning attention, q, k and v through silu):
//   S <- diag(a_t) S + k_t v_t^T,   o_t = S^T (q_scale q_t),   S [dk, dv] float32
// With D(s, t) the product of a channel's decays after s up to t and S_0 the state that a chunk of 64 tokens starts from:
//   P_ts = sum_i q_t k_s D(s, t)  (s <= t)      U = (k_s D(s, 64))^T V
//   O = (q_t D(0, t)) S_0 + P V                 S_64 = diag(D(0, 64)) S_0 + U
// so everything but one multiply-add a state element and chunk runs for all chunks side by side:
//   scan_chunk_state_kernel   P, U, the decayed q and D(0, 64) of every chunk
//   scan_chunk_carry_kernel   the state that every chunk starts from, in U's place
//   scan_chunk_out_kernel     O of every chunk
// No logarithm is taken of a decay: what lies between two tokens is a product of decays, which rounds like the walk does.  Sub-chunks of
// 16 tokens are related through the products at their edges, the tokens inside one as chunk_mma.cuh has it.
//
// U and O are products on the tensor cores.  q, k and v as projected are bfloat16 numbers and exact there; what is float32 (decayed
// q and k, P, S_0, anything that went through silu) goes in as the sum of three (chunk_mma.cuh).  A chunk with a number that is not finite
// among its q, k, v, decays or its S_0, or with a q or k beyond CHK_LARGE, is walked token by token, so that it does what the walk does.
//
// The walk in two passes over chunks of 128 (scan.cu) is bound by shared-memory reads and shuffles: a state element costs a token five
// instructions and a pass its own staging.  Measured beside it, with its kernel for the decays, L2 flushed, us: a decay a channel, 8 heads of
// 128 x 256, 2,048 tokens 79 / 277, 1,500 + 1,200 + 900 tokens 146 / 500, 8 x 128 tokens 56 / 181; 4 heads of 64 x 128 2,048 tokens 32 / 155.
// Constant decays behind silu, 8 heads of 128 x 256, 2,048 tokens 105 / 249; 4 heads of 64 x 128 34 / 91.  Of the 146 the states of the chunks
// take 62, the carry 21, the outputs 60: mma.sync takes 8.2 cycles a scheduler, and the outputs 120 of them a warp for 48 KB of operands
// that are split on the way.  (P by float32 sums, numbers loaded one by one and 32 decays a thread unrolled: 70 us for the states.)
#include "chunk_mma.cuh"

#define CHK_VB 64                          // value columns a turn of the state kernel
#define CHK_VPITCH (CHK_VB + 8)

struct ChunkArgs {
    const __nv_bfloat16 *q, *k, *v;
    long long q_stride, k_stride, v_stride;
    const float* gate;                     // [rows, heads * dk] logits or decays, or [heads] constants
    long long gate_stride;
    const __nv_bfloat16* gate_bias;        // [heads * dk] (logits)
    float* out; long long out_stride;
    uint8_t* state; long long state_stride, state_offset;
    const int *q_start, *q_len, *slot_ids;
    int heads, groups, dv, constant, gate_is_decay;
    int wide_qk, wide_gate;                // rows of q and k, of gate start on 16 bytes
    float q_scale, inv_tau;
    float *u, *qe, *p, *d;                 // blocks a (chunk, head): [dk][dv], [64][dk], [64][64], [dk]
    int* odd;                              // walked token by token
};

// The place of chunk c of sequence seq among all chunks of the step (a sequence of n rows takes ceil(n / 64) places, the next one starts
// at least so many further on).
__device__ __forceinline__ size_t chk_block(const ChunkArgs& a, int seq, int c, int h) {
    return (size_t)(a.q_start[seq] / CHK_C + seq + c) * a.heads + h;
}
__device__ __forceinline__ float chk_decay_of_logit(float z, float inv_tau) {
    return expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * inv_tau);
}
__device__ __forceinline__ float chk_decay(const ChunkArgs& a, int dk, int h, size_t row, int i) {
    if (a.constant) return a.gate[h];
    const float z = a.gate[row * a.gate_stride + (size_t)h * dk + i];
    return a.gate_is_decay ? z : chk_decay_of_logit(z + to_f32(a.gate_bias[(size_t)h * dk + i]), a.inv_tau);
}
template <bool SILU> __device__ __forceinline__ float chk_in(__nv_bfloat16 x) { return SILU ? silu_f32(to_f32(x)) : to_f32(x); }

// 64 tokens x 64 value columns as they come: 16 bytes a thread and turn, zeros past the sequence
__device__ __forceinline__ uint4 chk_load_v(const ChunkArgs& a, int h, int r0, int n, int col0, int idx) {
    const int r = idx >> 3, c = idx & 7;
    if (r >= n) return make_uint4(0, 0, 0, 0);
    return *reinterpret_cast<const uint4*>(a.v + (size_t)(r0 + r) * a.v_stride + (size_t)h * a.dv + col0 + c * 8);
}
// ... to shared memory, in one part (as they are) or three (after silu); rows of `pitch` elements, parts of `part` elements.  True: a number
// is not finite.
template <bool SILU>
__device__ __forceinline__ bool chk_store_v(__nv_bfloat16* dst, int pitch, int part, uint4 x, int idx) {
    const int r = idx >> 3, c = idx & 7;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    uint32_t top = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) top |= (w[e] & 0x7f807f80u) + 0x00800080u;
    __nv_bfloat16* at = dst + r * pitch + c * 8;
    if (!SILU) {
        *reinterpret_cast<uint4*>(at) = x;
    } else {
        uint32_t o[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            chk_split2(silu_f32(__uint_as_float(w[e] << 16)), silu_f32(__uint_as_float(w[e] & 0xffff0000u)), o[0][e], o[1][e], o[2][e]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(at + p * part) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
    }
    return (top & 0x80008000u) != 0;
}

// A chunk token by token, a thread a value column, the state in global memory: for numbers that are not finite.
template <bool SILU, bool OUT>
__device__ __noinline__ void chk_walk(const ChunkArgs& a, int dk, int h, int g, int r0, int n, float* S, int col0, int cols) {
    for (int jj = threadIdx.x; jj < cols; jj += CHK_THREADS) {
        const int j = col0 + jj;
        if (!OUT)
            for (int i = 0; i < dk; ++i) S[(size_t)i * a.dv + j] = 0.f;
        for (int t = 0; t < n; ++t) {
            const size_t row = (size_t)(r0 + t);
            const float v = chk_in<SILU>(a.v[row * a.v_stride + (size_t)h * a.dv + j]);
            float acc = 0.f;
            for (int i = 0; i < dk; ++i) {
                const float s = fmaf(chk_decay(a, dk, h, row, i), S[(size_t)i * a.dv + j], chk_in<SILU>(a.k[row * a.k_stride + (size_t)g * dk + i]) * v);
                S[(size_t)i * a.dv + j] = s;
                if (OUT) acc = fmaf(s, chk_in<SILU>(a.q[row * a.q_stride + (size_t)g * dk + i]) * a.q_scale, acc);
            }
            if (OUT) a.out[row * a.out_stride + (size_t)h * a.dv + j] = acc;
        }
    }
}

template <int DK, bool SILU> constexpr int chk_state_smem() {
    return (2 * CHK_C * (DK + 8) + 8 * DK) * 4 + (SILU ? 3 : 2) * CHK_C * CHK_VPITCH * 2;
}

// A CTA of eight warps owns a (chunk, head).  Everything is brought to shared memory 16 bytes a load, all loads in flight at once; a thread
// works a channel's decays out over one or two sub-chunks; P's rows of 16 are shared by two warps each; then a warp owns 16 rows of U, its
// operand (k decayed to the chunk's end) stays in its registers for all value columns.
template <int DK, bool SILU>
__global__ void __launch_bounds__(CHK_THREADS, 2)
scan_chunk_state_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int C = CHK_C, SUB = CHK_SUB, LD = DK + 8, NT = CHK_THREADS;
    constexpr int PV = SILU ? 3 : 1;
    extern __shared__ __align__(16) float chk_sm[];
    float* sQ = chk_sm;                                      // [C][LD]: decays; then q decayed from its sub-chunk's start, times CHK_UP
    float* sK = sQ + C * LD;                                 // [C][LD]: k, then decayed to its sub-chunk's end, times CHK_UP
    float* sT = sK + C * LD;                                 // [4][DK]: a sub-chunk's decays multiplied
    float* sI = sT + 4 * DK;                                 // [4][DK]: 1 / (that CHK_UP^2), 0 for a steep channel
    __nv_bfloat16* sV = (__nv_bfloat16*)(sI + 4 * DK);       // two buffers, or one of three parts
    static_assert(CHK_STEEP_FLOATS(DK) <= C * LD, "the steep channels are staged where q was");
    const int h = blockIdx.x, seq = blockIdx.y, c = blockIdx.z, tid = threadIdx.x;
    const int n = min(C, a.q_len[seq] - c * C), r0 = a.q_start[seq] + c * C;
    if (n <= 0) return;
    const int g = h / (a.heads / a.groups), dv = a.dv;
    const size_t block = chk_block(a, seq, c, h);
    const int warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lq = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    pdl_wait();
    bool bad = false;
    uint4 vx[2], qx[C * DK / 8 / NT];
    const int run = tid % (DK / 8) * 8, row8 = tid / (DK / 8);                   // this thread's channels of a row of q and k, its first row
    const int ch4 = tid % (DK / 4) * 4, row4 = tid / (DK / 4);                   // of decays
    constexpr int STEP8 = NT * 8 / DK, STEP4 = NT * 4 / DK;
    {
        uint4 kx[C * DK / 8 / NT];
        float4 zx[C * DK / 4 / NT];
#pragma unroll
        for (int w = 0; w < C * DK / 4 / NT; ++w) {
            const int t = row4 + w * STEP4;
            zx[w] = a.constant || t >= n ? make_float4(0.f, 0.f, 0.f, 0.f) : chk_load4(a.gate + (size_t)(r0 + t) * a.gate_stride + (size_t)h * DK + ch4, a.wide_gate);
        }
#pragma unroll
        for (int w = 0; w < C * DK / 8 / NT; ++w) {
            const int t = row8 + w * STEP8;
            kx[w] = t < n ? chk_load8(a.k + (size_t)(r0 + t) * a.k_stride + (size_t)g * DK + run, a.wide_qk) : make_uint4(0, 0, 0, 0);
            qx[w] = t < n ? chk_load8(a.q + (size_t)(r0 + t) * a.q_stride + (size_t)g * DK + run, a.wide_qk) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) vx[w] = chk_load_v(a, h, r0, n, 0, tid + w * NT);
#pragma unroll
        for (int w = 0; w < C * DK / 4 / NT; ++w) *reinterpret_cast<float4*>(sQ + (row4 + w * STEP4) * LD + ch4) = zx[w];
#pragma unroll
        for (int w = 0; w < C * DK / 8 / NT; ++w) *reinterpret_cast<uint4*>(sK + (row8 + w * STEP8) * LD + run) = kx[w];       // (widened below)
    }
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (!a.constant && !a.gate_is_decay)
#pragma unroll
        for (int e = 0; e < 4; ++e) bias[e] = to_f32(a.gate_bias[(size_t)h * DK + ch4 + e]);
#pragma unroll 2
    for (int t = row4; t < C; t += STEP4) {                  // a loop: its body is the longest code of the kernel
        float4* at = reinterpret_cast<float4*>(sQ + t * LD + ch4);
        const float4 v = *at;
        float d[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (a.constant) d[e] = a.gate[h];
            else if (!a.gate_is_decay) d[e] = chk_decay_of_logit(d[e] + bias[e], a.inv_tau);
            if (t >= n) d[e] = 1.f;
            bad |= chk_not_finite(d[e]);
        }
        *at = make_float4(d[0], d[1], d[2], d[3]);
    }
    auto widen = [&](uint4 x, float* y, float scale) {
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            y[2 * e] = __uint_as_float(w[e] << 16);
            y[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (SILU) y[e] = silu_f32(y[e]);
            bad |= !(fabsf(y[e] * scale) <= CHK_LARGE);
        }
    };
#pragma unroll 1
    for (int t = row8; t < C; t += STEP8) {
        float* at = sK + t * LD + run;
        float y[8];
        widen(*reinterpret_cast<const uint4*>(at), y, 1.f);
        *reinterpret_cast<float4*>(at) = make_float4(y[0], y[1], y[2], y[3]);
        *reinterpret_cast<float4*>(at + 4) = make_float4(y[4], y[5], y[6], y[7]);
    }
    __syncthreads();
    bool any_steep = false;
#pragma unroll 1
    for (int w = tid; w < 4 * DK; w += NT) {                 // a (sub-chunk, channel)
        float *d = sQ + w / DK * SUB * LD + w % DK, *k = sK + w / DK * SUB * LD + w % DK;
        any_steep |= chk_decays<LD, false>(d, k, nullptr, sT + w, sI + w);
    }
    any_steep = __syncthreads_or(any_steep);
#pragma unroll
    for (int w = 0; w < C * DK / 8 / NT; ++w) {
        float* at = sQ + (row8 + w * STEP8) * LD + run;
        float y[8], e[8];
        widen(qx[w], y, a.q_scale);
        *reinterpret_cast<float4*>(e) = *reinterpret_cast<const float4*>(at);
        *reinterpret_cast<float4*>(e + 4) = *reinterpret_cast<const float4*>(at + 4);
#pragma unroll
        for (int x = 0; x < 8; ++x) y[x] *= a.q_scale * (e[x] * CHK_UP);
        *reinterpret_cast<float4*>(at) = make_float4(y[0], y[1], y[2], y[3]);
        *reinterpret_cast<float4*>(at + 4) = make_float4(y[4], y[5], y[6], y[7]);
    }
    __syncthreads();
    // the rows of 16 by two warps each, 8 keys of every sub-chunk a warp; rows with more sub-chunks share a scheduler with ones of fewer
    const int J = warp < 4 ? warp : 7 - warp, tile = warp >> 2;
    float P[4][1][2][4];
    chk_scores<DK, LD, 1>(sQ + J * SUB * LD, sK, sT, sI, J, tile, P);
    float* gQ = a.qe + block * (C * DK);
#pragma unroll 4
    for (int idx = tid * 4; idx < C * DK; idx += NT * 4) {   // q decayed from the chunk's start
        const int t = idx / DK, i = idx % DK;
        float x[4];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(sQ + t * LD + i);
        for (int m = t / SUB - 1; m >= 0; --m)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] *= sT[m * DK + i + e];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] *= 1.f / CHK_UP;
        *reinterpret_cast<float4*>(gQ + idx) = make_float4(x[0], x[1], x[2], x[3]);
    }
    if (any_steep) {
        __syncthreads();                                     // q has been used
        chk_steep<DK, false>(sQ, sI, n, [&](int t, int i) { return chk_in<SILU>(a.q[(size_t)(r0 + t) * a.q_stride + (size_t)g * DK + i]) * a.q_scale; },
                             [&](int t, int i) { return chk_in<SILU>(a.k[(size_t)(r0 + t) * a.k_stride + (size_t)g * DK + i]); },
                             [&](int t, int i) { return chk_decay(a, DK, h, (size_t)(r0 + t), i); },
                             [&](int sub, const float* p, const float*) {
                                 if (sub == J)
#pragma unroll
                                     for (int e = 0; e < 4; ++e) P[0][0][0][e] += p[(lg + (e >> 1) * 8) * 17 + tile * 8 + lq + (e & 1)];
                             });
    }
    float* gP = a.p + block * (C * C);
#pragma unroll
    for (int d = 0; d < 4; ++d)
        if (d <= J)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = lg + e * 8, s = tile * 8 + lq;
                float x = P[d][0][0][2 * e], y = P[d][0][0][2 * e + 1];
                if (d == 0) { x = s <= t ? x : 0.f; y = s + 1 <= t ? y : 0.f; }      // later tokens are left out, whatever their products are
                *reinterpret_cast<float2*>(gP + (J * SUB + t) * C + (J - d) * SUB + s) = make_float2(x, y);
            }
    if (tid < DK) a.d[block * DK + tid] = sT[tid] * sT[DK + tid] * sT[2 * DK + tid] * sT[3 * DK + tid];
    // U: the warp's 16 rows, k decayed to the chunk's end in three parts
    constexpr int MT = DK / 16, NW = 8 / MT, TILES = CHK_VB / 8 / NW;      // warps that share 16 rows, tiles of 8 columns a warp
    const int m0 = warp % MT * 16, t0 = warp / MT * TILES;
    uint32_t ka[4][3][4];
    {
        float tail[2] = {1.f / CHK_UP, 1.f / CHK_UP};
#pragma unroll
        for (int ks = 3; ks >= 0; --ks) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {                    // rows lg + (e & 1) * 8, tokens lq + (e >> 1) * 8 and the next
                const int i = m0 + lg + (e & 1) * 8;
                const float* at = sK + (ks * SUB + lq + (e >> 1) * 8) * LD + i;
                chk_split2(at[0] * tail[e & 1], at[LD] * tail[e & 1], ka[ks][0][e], ka[ks][1][e], ka[ks][2][e]);
            }
            tail[0] *= sT[ks * DK + m0 + lg];
            tail[1] *= sT[ks * DK + m0 + lg + 8];
        }
    }
    float* gU = a.u + block * ((size_t)DK * dv);
    const int blocks = dv / CHK_VB;
    for (int b = 0; b < blocks; ++b) {
        __nv_bfloat16* buf = SILU ? sV : sV + (b & 1) * (C * CHK_VPITCH);
        if (SILU) __syncthreads();                           // the parts before have been read
#pragma unroll
        for (int w = 0; w < 2; ++w) bad |= chk_store_v<SILU>(buf, CHK_VPITCH, C * CHK_VPITCH, vx[w], tid + w * NT);
        if (b + 1 < blocks)
#pragma unroll
            for (int w = 0; w < 2; ++w) vx[w] = chk_load_v(a, h, r0, n, (b + 1) * CHK_VB, tid + w * NT);
        __syncthreads();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float acc[TILES / 2][2][4];                      // the products of the first parts, and the small ones
#pragma unroll
            for (int x = 0; x < TILES / 2; ++x)
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[x][e >> 2][e & 3] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                for (int pr = 0; pr < TILES / 4; ++pr) {
                    uint32_t vb[PV][4];
#pragma unroll
                    for (int p = 0; p < PV; ++p)
                        chk_ldm4t(vb[p], chk_u32(buf + p * (C * CHK_VPITCH) + (ks * SUB + (lm & 1) * 8 + lr) * CHK_VPITCH + (t0 + half * TILES / 2) * 8 + pr * 16 + (lm >> 1) * 8));
                    CHK_PAIRS(3, PV, pa, pb) {
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (pa + pb == 0) chk_mma_sum<true>(acc[2 * pr + t], ka[ks][pa], vb[pb][2 * t], vb[pb][2 * t + 1]);
                            else chk_mma_sum<false>(acc[2 * pr + t], ka[ks][pa], vb[pb][2 * t], vb[pb][2 * t + 1]);
                    }
                }
            float* at = gU + (size_t)(m0 + lg) * dv + b * CHK_VB + (t0 + half * TILES / 2) * 8 + lq;
#pragma unroll
            for (int x = 0; x < TILES / 2; ++x) {
                const float (*v)[4] = acc[x];
                *reinterpret_cast<float2*>(at + x * 8) = make_float2(v[0][0] + v[1][0], v[0][1] + v[1][1]);
                *reinterpret_cast<float2*>(at + (size_t)8 * dv + x * 8) = make_float2(v[0][2] + v[1][2], v[0][3] + v[1][3]);
            }
        }
    }
    bad = __syncthreads_or(bad);
    if (bad) chk_walk<SILU, false>(a, DK, h, g, r0, n, gU, 0, dv);
    if (tid == 0) a.odd[block] = bad;
    pdl_trigger();
}

// The state that every chunk starts from: four neighbouring value columns a thread, chunk after chunk, eight chunks' numbers asked for
// before any of them is used.
template <int DK>
__global__ void __launch_bounds__(256)
scan_chunk_carry_kernel(const __grid_constant__ ChunkArgs a) {
    pdl_trigger();
    const int seq = blockIdx.y, per_head = DK * a.dv / 4;
    const int idx = blockIdx.x * 256 + threadIdx.x;
    const int n = a.q_len[seq];
    if (idx >= a.heads * per_head || n <= 0) return;
    const int n_chunks = (n + CHK_C - 1) / CHK_C, h = idx / per_head, rest = idx - h * per_head, i = rest * 4 / a.dv;
    float4* at = (float4*)(a.state + (size_t)a.slot_ids[seq] * a.state_stride + a.state_offset) + idx;
    pdl_wait();
    const size_t block0 = chk_block(a, seq, 0, h);
    float4* u = (float4*)a.u + block0 * per_head + rest;
    const float* d = a.d + block0 * DK + i;
    const size_t u_step = (size_t)a.heads * per_head, d_step = (size_t)a.heads * DK;
    float4 S = *at;
    constexpr int B = 8;
    for (int c0 = 0; c0 < n_chunks; c0 += B) {
        float4 uu[B];
        float dd[B];
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (c0 + j < n_chunks) {
                uu[j] = u[(c0 + j) * u_step];
                dd[j] = d[(c0 + j) * d_step];
            }
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (c0 + j < n_chunks) {
                u[(c0 + j) * u_step] = S;
                S.x = fmaf(dd[j], S.x, uu[j].x);
                S.y = fmaf(dd[j], S.y, uu[j].y);
                S.z = fmaf(dd[j], S.z, uu[j].z);
                S.w = fmaf(dd[j], S.w, uu[j].w);
            }
    }
    *at = S;
}

// A CTA owns 64 tokens x NB value columns of a (chunk, head).
template <int DK, bool SILU, int NB>
__global__ void __launch_bounds__(CHK_THREADS, 2)
scan_chunk_out_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int C = CHK_C, NT = CHK_THREADS;
    extern __shared__ __align__(16) float chk_sm[];
    pdl_trigger();
    const int cols = a.dv / NB;
    const int h = blockIdx.x, seq = blockIdx.y, c = blockIdx.z / cols, col0 = (blockIdx.z - c * cols) * NB, tid = threadIdx.x;
    const int n = min(C, a.q_len[seq] - c * C), r0 = a.q_start[seq] + c * C;
    if (n <= 0) return;
    const size_t block = chk_block(a, seq, c, h);
    pdl_wait();
    float* S = a.u + block * ((size_t)DK * a.dv);
    constexpr int VP = NB + 8;
    const int lane = tid & 31, lr = lane & 7, lm = lane >> 3, cw = chk_out_col<NB>();
    const float* sp = S + (size_t)((lane & 3) * 2) * a.dv + col0 + cw + (lane >> 2);
    const bool odd = chk_outputs<DK, SILU ? 3 : 1, NB, true>(
        chk_sm, a.qe + block * (C * DK), a.p + block * (C * C), a.odd[block] != 0,
        [&](float* x, int ks) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* at = sp + (size_t)(ks * 16 + (e & 1) + (e >> 1) * 8) * a.dv;
                x[e] = at[0];
                x[4 + e] = at[8];
            }
        },
        [&](__nv_bfloat16* v) {
#pragma unroll
            for (int w = 0; w < NB / 32; ++w) {
                const int idx = tid + (w & 1) * NT, b = (w >> 1) * 64;
                chk_store_v<SILU>(v + b, VP, C * VP, chk_load_v(a, h, r0, n, col0 + b, idx), idx);
            }
        },
        [&](uint32_t (*b)[4], int ks, const __nv_bfloat16* v) {
#pragma unroll
            for (int p = 0; p < (SILU ? 3 : 1); ++p) chk_ldm4t(b[p], chk_u32(v + p * C * VP + (ks * 16 + (lm & 1) * 8 + lr) * VP + cw + (lm >> 1) * 8));
        },
        [&](int t, int col, float x, float y) {
            if (t < n) *reinterpret_cast<float2*>(a.out + (size_t)(r0 + t) * a.out_stride + (size_t)h * a.dv + col0 + col) = make_float2(x, y);
        });
    if (odd) chk_walk<SILU, true>(a, DK, h, h / (a.heads / a.groups), r0, n, S, col0, NB);
}

static long long chk_blocks(int rows, int n_seqs, int heads) { return ((long long)rows / CHK_C + n_seqs + 1) * heads; }

// Floats of scratch that a step needs.
extern "C" long long braid_scan_chunk_work_floats(int rows, int n_seqs, int heads, int dk, int dv) {
    return chk_blocks(rows, n_seqs, heads) * ((long long)dk * dv + CHK_C * dk + CHK_C * CHK_C + dk + 1);
}

template <int DK, bool SILU, int NB>
static int launch_scan_chunk(const ChunkArgs& a, int n_seqs, int chunks, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(scan_chunk_state_kernel<DK, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, chk_state_smem<DK, SILU>());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(scan_chunk_out_kernel<DK, SILU, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (chk_out_smem<DK, (SILU ? 3 : 1) * CHK_C * (NB + 8) * 2>()));
        if (e != cudaSuccess) { braid_set_error("scan_chunk: cannot reserve shared memory: %s", cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    braid_launch(scan_chunk_state_kernel<DK, SILU>, dim3(a.heads, n_seqs, chunks), dim3(CHK_THREADS), (size_t)chk_state_smem<DK, SILU>(), s, a);
    braid_launch(scan_chunk_carry_kernel<DK>, dim3((unsigned)(((long long)a.heads * DK * a.dv / 4 + 255) / 256), n_seqs), dim3(256), 0, s, a);
    braid_launch(scan_chunk_out_kernel<DK, SILU, NB>, dim3(a.heads, n_seqs, chunks * (a.dv / NB)), dim3(CHK_THREADS), (size_t)(chk_out_smem<DK, (SILU ? 3 : 1) * CHK_C * (NB + 8) * 2>()), s, a);
    BRAID_LAUNCH_CHECK();
}

// bfloat16 rows on 16 bytes; dk 64 or 128, dv a multiple of 64.  `constant`: gate holds one decay a head; else [rows, heads * dk] logits
// (with their bias and inv_tau) or, with gate_is_decay, decays.  act_silu: q, k and v go through silu.
extern "C" int braid_scan_chunk(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                                const float* gate, long long gate_stride, const void* gate_bias, float* out, long long out_stride,
                                void* state, long long state_stride, long long state_offset, const int* q_start, const int* q_len,
                                const int* slot_ids, int rows, int n_seqs, int max_q_len, int heads, int groups, int dk, int dv,
                                float q_scale, float inv_tau, int constant, int gate_is_decay, int act_silu, float* work,
                                long long work_floats, void* stream) {
    if (n_seqs <= 0 || rows <= 0 || max_q_len <= 0) return BRAID_OK;
    if (heads <= 0 || groups <= 0 || heads % groups) BRAID_REFUSE("scan_chunk: %d heads do not divide into %d groups", heads, groups);
    if ((dk != 64 && dk != 128) || dv <= 0 || dv % 64) BRAID_REFUSE("scan_chunk: built for keys of 64 or 128 and values in multiples of 64, not %d x %d", dk, dv);
    if (((uintptr_t)v & 15) || v_stride % 8) BRAID_REFUSE("scan_chunk: rows of v must start on 16 bytes");
    if (((uintptr_t)out & 7) || out_stride % 2 || !state || (((uintptr_t)state | (uintptr_t)state_offset | (uintptr_t)state_stride) & 15))
        BRAID_REFUSE("scan_chunk: results must start on 8 bytes and the state on 16");
    if (!gate || (!constant && !gate_is_decay && !gate_bias)) BRAID_REFUSE("scan_chunk: the decays are missing");
    if (act_silu && !constant) BRAID_REFUSE("scan_chunk: silu on what is given goes with a constant decay a head");
    const long long need = braid_scan_chunk_work_floats(rows, n_seqs, heads, dk, dv);
    if (!work || need > work_floats || ((uintptr_t)work & 15)) BRAID_REFUSE("scan_chunk: needs %lld floats of scratch on 16 bytes, it was given %lld", need, work_floats);
    const int chunks = (max_q_len + CHK_C - 1) / CHK_C;
    if (n_seqs > 65535 || (long long)chunks * (dv / 64) > 65535 || (long long)heads * dk * dv > 0x7fffffffLL) BRAID_REFUSE("scan_chunk: the step exceeds the grid limits");
    const long long blocks = chk_blocks(rows, n_seqs, heads);
    using B = const __nv_bfloat16*;
    ChunkArgs a{(B)q, (B)k, (B)v, q_stride, k_stride, v_stride, gate, gate_stride, (B)gate_bias, out, out_stride, (uint8_t*)state,
                state_stride, state_offset, q_start, q_len, slot_ids, heads, groups, dv, constant, gate_is_decay,
                (((uintptr_t)q | (uintptr_t)k) & 15) == 0 && q_stride % 8 == 0 && k_stride % 8 == 0, ((uintptr_t)gate & 15) == 0 && gate_stride % 4 == 0, q_scale, inv_tau};
    a.u = work;
    a.qe = a.u + blocks * dk * dv;
    a.p = a.qe + blocks * CHK_C * dk;
    a.d = a.p + blocks * CHK_C * CHK_C;
    a.odd = (int*)(a.d + blocks * dk);
    cudaStream_t s = (cudaStream_t)stream;
    if (act_silu) return dk == 64 ? launch_scan_chunk<64, true, 64>(a, n_seqs, chunks, s) : launch_scan_chunk<128, true, 64>(a, n_seqs, chunks, s);
    if (dv % 128) return dk == 64 ? launch_scan_chunk<64, false, 64>(a, n_seqs, chunks, s) : launch_scan_chunk<128, false, 64>(a, n_seqs, chunks, s);
    return dk == 64 ? launch_scan_chunk<64, false, 128>(a, n_seqs, chunks, s) : launch_scan_chunk<128, false, 128>(a, n_seqs, chunks, s);
}
