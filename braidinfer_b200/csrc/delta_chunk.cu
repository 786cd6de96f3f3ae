// The chunks of delta.cu's rule for key sizes up to 128 (beyond: delta_intra_kernel, delta_state_kernel and delta_out_kernel there): the same
// equations with the products on mma.sync, float32 operands as sums of three bfloat16 numbers (chunk_mma.cuh).
//   delta_rows_kernel    P, the decayed queries, and W, U0 and the decayed keys (as bfloat16 parts where they are operands) of every chunk
//   delta_chain_kernel   chunk after chunk: U, and the state every chunk starts from
//   delta_outputs_kernel O of every chunk
// (I + diag(beta) A) X = diag(beta) R is solved 16 tokens at a time, X_J = T_J (beta R_J - sum_I<J (beta A)_JI X_I) with T_J the inverse of
// the block on the diagonal, X transposed: a warp's 16 columns of X are accumulators of one product and the operand of the next.
// The chain is what a prompt waits for.  Two warps of it own 16 value columns, each half of the keys, and keep their transposed state in
// their accumulators, which are the operand of S^T W^T as U^T is of U^T K: the state never passes through shared memory, only the two
// halves of S^T W^T meet there.  U and the states lie in memory as the lanes hold them, [16 value columns][16 tokens or keys][lane][8], which
// is how the outputs' products want them too.
// A token's numbers that are not finite may reach back inside its own block of 16 (zeros of the triangles times them), as they did in the sums on
// the ordinary pipes; never to the tokens of earlier blocks, other heads or sequences.
// Measured, 16 heads of 128 x 256, 1,777 + 1,244 tokens, us, beside float32 sums on the ordinary pipes: rows 171 / 272, chain 193 / 265,
// outputs 94 / 142.  The chain is bound by mma.sync (768 a scheduler and chunk at 8.2 cycles are 6,300 of its 10,500 cycles), the rows by the
// dependent products of the solve.
#include "delta.cuh"
#include "chunk_mma.cuh"

#define DLC_COLS 64                        // value columns a CTA of the chain and of the outputs
#define DLC_APITCH (CHK_C + 8)
#define DLC_TPITCH 24

// A's blocks below the diagonal in three parts, the inverses in three parts, the blocks on the diagonal
constexpr int dlc_solve_bytes() { return 3 * CHK_C * DLC_APITCH * 2 + 3 * CHK_C * DLC_TPITCH * 2 + CHK_C * 17 * 4; }
template <int DK> constexpr int dlc_first_bytes() { return CHK_C * (DK + 8) * 4 > dlc_solve_bytes() ? CHK_C * (DK + 8) * 4 : dlc_solve_bytes(); }
template <int DK> constexpr int dlc_rows_smem() { return dlc_first_bytes<DK>() + (2 * CHK_C * (DK + 8) + 8 * DK + CHK_C) * 4; }
template <int DK> constexpr int dlc_chain_smem() { return 2 * 2 * 3 * CHK_C * DK * 2 + 8 * CHK_C * 16 * 4 + 2 * DK * 4; }

// Everything is brought to shared memory 16 bytes a load; a thread works a channel's decays out over one or two sub-chunks; a warp owns 16 rows
// of A or of P; then 16 columns of X.
template <typename T, int DK>
__global__ void __launch_bounds__(CHK_THREADS, 2)
delta_rows_kernel(const __grid_constant__ DeltaArgs a) {
    constexpr int C = CHK_C, SUB = CHK_SUB, LD = DK + 8, NT = CHK_THREADS;
    extern __shared__ __align__(128) uint8_t dlc_bytes[];
    float* sQ = (float*)dlc_bytes;                           // [C][LD]: decays, q decayed from its sub-chunk's start (times CHK_UP); then the solve's operands:
    __nv_bfloat16* sA = (__nv_bfloat16*)dlc_bytes;           //   3 x [C][DLC_APITCH]: -beta_t A_ts
    __nv_bfloat16* sX = sA + 3 * C * DLC_APITCH;             //   3 x [C][DLC_TPITCH]: the inverses of the diagonal's blocks, side by side
    float* sL = (float*)(sX + 3 * C * DLC_TPITCH);           //   [C][17]: beta_t A_ts of the diagonal's blocks
    float* sF = (float*)(dlc_bytes + dlc_first_bytes<DK>()); // [C][LD]: k decayed from its sub-chunk's start (times CHK_UP), then from the chunk's
    float* sK = sF + C * LD;                                 // [C][LD]: k decayed to its sub-chunk's end, times CHK_UP
    float* sT = sK + C * LD;                                 // [4][DK]: a sub-chunk's decays multiplied
    float* sI = sT + 4 * DK;                                 // [4][DK]: 1 / (that CHK_UP^2), 0 for a steep channel
    float* sB = sI + 4 * DK;                                 // beta
    static_assert(CHK_STEEP_FLOATS(DK) * 4 <= dlc_first_bytes<DK>(), "the steep channels are staged where q was");
    const int h = blockIdx.x, seq = blockIdx.y, c = blockIdx.z, tid = threadIdx.x;
    const int n = min(C, a.q_len[seq] - c * C), r0 = a.q_start[seq] + c * C;
    if (n <= 0) return;
    const int dk = a.dk, dv = a.dv, g = h / (a.heads / a.groups), dvp = a.tiles * DLC_COLS;
    const size_t block = delta_block(a, seq, c, h);
    const float rate = a.rate[h];
    pdl_wait();
    const int warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lq = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    const int ch4 = tid % (DK / 4) * 4, row4 = tid / (DK / 4);       // this thread's channels of a row, its first row
    constexpr int N4 = C * DK / 4 / NT, STEP4 = NT * 4 / DK;
    // (channels past dk read as zeros; a run of four lies on one side of dk or the numbers are taken one by one)
    auto four = [&](const float* p, bool wide, int t) {
        if (t >= n || ch4 >= dk) return make_float4(0.f, 0.f, 0.f, 0.f);
        if (ch4 + 4 <= dk) return chk_load4(p, wide);
        return make_float4(p[0], ch4 + 1 < dk ? p[1] : 0.f, ch4 + 2 < dk ? p[2] : 0.f, 0.f);
    };
    float4 qx[N4];
    {
        float4 kx[N4], zx[N4];
#pragma unroll
        for (int w = 0; w < N4; ++w) {
            const int t = row4 + w * STEP4;
            zx[w] = four(a.z + (size_t)(r0 + t) * a.z_stride + (size_t)h * dk + ch4, a.wide_z, t);
            kx[w] = four(a.k + (size_t)(r0 + t) * a.k_stride + (size_t)g * dk + ch4, a.wide_qk, t);
        }
#pragma unroll
        for (int w = 0; w < N4; ++w) {
            const int t = row4 + w * STEP4;
            qx[w] = four(a.q + (size_t)(r0 + t) * a.q_stride + (size_t)g * dk + ch4, a.wide_qk, t);
        }
#pragma unroll
        for (int w = 0; w < N4; ++w) {
            *reinterpret_cast<float4*>(sQ + (row4 + w * STEP4) * LD + ch4) = zx[w];
            *reinterpret_cast<float4*>(sK + (row4 + w * STEP4) * LD + ch4) = kx[w];
        }
    }
    if (tid < C) sB[tid] = tid < n ? delta_sigmoid(to_f32(((const T*)a.b)[(size_t)(r0 + tid) * a.b_stride + h])) : 0.f;
    float bias[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) bias[e] = ch4 + e < dk ? a.bias[(size_t)h * dk + ch4 + e] : 0.f;
#pragma unroll 2
    for (int t = row4; t < C; t += STEP4) {                  // a loop: its body is the longest code of the kernel
        float4* at = reinterpret_cast<float4*>(sQ + t * LD + ch4);
        const float4 v = *at;
        float d[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] = t < n && ch4 + e < dk ? delta_decay(d[e] + bias[e], rate) : 1.f;
        *at = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
    bool steep = false;
#pragma unroll 1
    for (int w = tid; w < 4 * DK; w += NT) {                 // a (sub-chunk, channel)
        const int at = w / DK * SUB * LD + w % DK;
        steep |= chk_decays<LD, true>(sQ + at, sK + at, sF + at, sT + w, sI + w);
    }
    steep = __syncthreads_or(steep);
#pragma unroll
    for (int w = 0; w < N4; ++w) {
        float4* at = reinterpret_cast<float4*>(sQ + (row4 + w * STEP4) * LD + ch4);
        const float4 e = *at;
        *at = make_float4(qx[w].x * (e.x * CHK_UP), qx[w].y * (e.y * CHK_UP), qx[w].z * (e.z * CHK_UP), qx[w].w * (e.w * CHK_UP));
    }
    __syncthreads();
    // P's rows of 16 by the first four warps, A's by the others: rows with more sub-chunks share a scheduler with ones of fewer
    const bool is_p = warp < 4;
    const int J = is_p ? warp : 7 - warp;
    float M[4][2][2][4];
    chk_scores<DK, LD, 2>((is_p ? sQ : sF) + J * SUB * LD, sK, sT, sI, J, 0, M);
    __syncthreads();                                         // F is decayed further in place
    // the operands: q decayed from the chunk's start, k to its end (three parts), k from its start
    float* gQ = a.qd + block * (C * DK);
    __nv_bfloat16 *gK = a.kp + block * (3 * C * DK), *gW = a.wp + block * (3 * C * DK);
#pragma unroll 1
    for (int idx = tid * 4; idx < C * DK; idx += NT * 4) {
        const int t = idx / DK, i = idx % DK, J = t / SUB;
        float x[4], f[4], k[4], m[4];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(sQ + t * LD + i);
        *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(sF + t * LD + i);
        *reinterpret_cast<float4*>(k) = *reinterpret_cast<const float4*>(sK + t * LD + i);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if (w == J) continue;
            *reinterpret_cast<float4*>(m) = *reinterpret_cast<const float4*>(sT + w * DK + i);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (w < J) { x[e] *= m[e]; f[e] *= m[e]; }
                else k[e] *= m[e];
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) { x[e] *= 1.f / CHK_UP; f[e] *= 1.f / CHK_UP; k[e] *= 1.f / CHK_UP; }
        *reinterpret_cast<float4*>(gQ + idx) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(sF + t * LD + i) = make_float4(f[0], f[1], f[2], f[3]);
        chk_store_split4(gK + idx, C * DK, make_float4(k[0], k[1], k[2], k[3]));
    }
    if (tid < DK) a.gc[block * DK + tid] = sT[tid] * sT[DK + tid] * sT[2 * DK + tid] * sT[3 * DK + tid];
    __syncthreads();                                         // q has been used
    if (steep)
        chk_steep<DK, true>(sQ, sI, n, [&](int t, int i) { return i < dk ? a.q[(size_t)(r0 + t) * a.q_stride + (size_t)g * dk + i] : 0.f; },
                            [&](int t, int i) { return i < dk ? a.k[(size_t)(r0 + t) * a.k_stride + (size_t)g * dk + i] : 0.f; },
                            [&](int t, int i) { return i < dk ? delta_decay(a.z[(size_t)(r0 + t) * a.z_stride + (size_t)h * dk + i] + a.bias[(size_t)h * dk + i], rate) : 1.f; },
                            [&](int sub, const float* p, const float* q) {
                                if (sub == J)
#pragma unroll
                                    for (int x = 0; x < 2; ++x)
#pragma unroll
                                        for (int e = 0; e < 4; ++e) M[0][x][0][e] += (is_p ? p : q)[(lg + (e >> 1) * 8) * 17 + x * 8 + lq + (e & 1)];
                            });
    float* gP = a.p + block * (C * C);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        if (d > J) continue;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = lg + e * 8, t = J * SUB + r, s = x * 8 + lq, at = (J - d) * SUB + s;
                float v = M[d][x][0][2 * e], w = M[d][x][0][2 * e + 1];
                if (is_p) {
                    if (d == 0) { v = s <= r ? v : 0.f; w = s + 1 <= r ? w : 0.f; }
                    *reinterpret_cast<float2*>(gP + t * C + at) = make_float2(v, w);
                    continue;
                }
                const float beta = sB[t];
                if (d == 0) {
                    sL[t * 17 + s] = s < r ? beta * v : 0.f;
                    sL[t * 17 + s + 1] = s + 1 < r ? beta * w : 0.f;
                } else {
                    uint32_t y[3];
                    chk_split2(-beta * v, -beta * w, y[0], y[1], y[2]);
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(sA + (p * C + t) * DLC_APITCH + at) = y[p];
                }
            }
    }
    __syncthreads();
    if (tid < C) {                                           // a thread a column of an inverse: forward substitution
        const int J = tid / SUB, s = tid % SUB;
        const float* L = sL + J * SUB * 17;
        float x[SUB];
#pragma unroll
        for (int t = 0; t < SUB; ++t) {
            float acc = t == s ? 1.f : 0.f;
#pragma unroll
            for (int r = 0; r < t; ++r) acc = fmaf(-L[t * 17 + r], x[r], acc);
            x[t] = acc;
        }
#pragma unroll
        for (int t = 0; t < SUB; ++t) {
            uint32_t w[3];
            chk_split2(x[t], 0.f, w[0], w[1], w[2]);
#pragma unroll
            for (int p = 0; p < 3; ++p) reinterpret_cast<uint16_t*>(sX)[(p * C + J * SUB + t) * DLC_TPITCH + s] = (uint16_t)w[p];
        }
    }
    __syncthreads();
    float* gU = a.u + block * (size_t)(C * dvp);
#pragma unroll 1
    for (int grp = warp; grp < (DK + dvp) / 16; grp += 8) {
        const bool is_w = grp < DK / 16;
        const int col = is_w ? grp * 16 + lg : grp * 16 - DK + lg;       // and col + 8
        uint32_t xa[3][3][4];                                // X^T of the 16 tokens of block I, in parts
        float next[2][4];                                    // the right sides of the block to come: columns col (+ 8), tokens x * 8 + lq (+ 1)
        auto fetch = [&](int J) {
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = J * SUB + x * 8 + lq + (e & 1), at = col + (e >> 1) * 8;
                    next[x][e] = 0.f;
                    if (is_w) next[x][e] = sF[t * LD + at];
                    else if (t < n && at < dv) next[x][e] = a.v[(size_t)(r0 + t) * a.v_stride + (size_t)h * dv + at];
                }
        };
        fetch(0);
#pragma unroll
        for (int J = 0; J < 4; ++J) {
            float y[2][2][4];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    y[x][0][e] = next[x][e] * sB[J * SUB + x * 8 + lq + (e & 1)];
                    y[x][1][e] = 0.f;
                }
            if (J < 3) fetch(J + 1);
#pragma unroll
            for (int I = 0; I < J; ++I) {
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) chk_ldm4(b[p], chk_u32(sA + (p * C + J * SUB + (lm >> 1) * 8 + lr) * DLC_APITCH + I * SUB + (lm & 1) * 8));
                CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                    for (int x = 0; x < 2; ++x)
                        if (pa + pb == 0) chk_mma_sum<true>(y[x], xa[I][pa], b[pb][2 * x], b[pb][2 * x + 1]);
                        else chk_mma_sum<false>(y[x], xa[I][pa], b[pb][2 * x], b[pb][2 * x + 1]);
                }
            }
            uint32_t ya[3][4], b[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float (*v)[4] = y[e >> 1];
                const int f = (e & 1) * 2;
                chk_split2(v[0][f] + v[1][f], v[0][f + 1] + v[1][f + 1], ya[0][e], ya[1][e], ya[2][e]);
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) chk_ldm4(b[p], chk_u32(sX + (p * C + J * SUB + (lm >> 1) * 8 + lr) * DLC_TPITCH + (lm & 1) * 8));
            float z[2][2][4];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 8; ++e) z[x][e >> 2][e & 3] = 0.f;
            CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                for (int x = 0; x < 2; ++x)
                    if (pa + pb == 0) chk_mma_sum<true>(z[x], ya[pa], b[pb][2 * x], b[pb][2 * x + 1]);
                    else chk_mma_sum<false>(z[x], ya[pa], b[pb][2 * x], b[pb][2 * x + 1]);
            }
            if (!is_w) {
                float4* at = reinterpret_cast<float4*>(gU) + ((size_t)((grp - DK / 16) * 4 + J) * 32 + lane) * 2;
#pragma unroll
                for (int x = 0; x < 2; ++x)
                    at[x] = make_float4(z[x][0][0] + z[x][1][0], z[x][0][1] + z[x][1][1], z[x][0][2] + z[x][1][2], z[x][0][3] + z[x][1][3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {                    // columns col + (e & 1) * 8, tokens t and t + 1
                const float (*v)[4] = z[e >> 1];
                const int f = (e & 1) * 2, t = J * SUB + (e >> 1) * 8 + lq, at = col + (e & 1) * 8;
                const float x0 = v[0][f] + v[1][f], x1 = v[0][f + 1] + v[1][f + 1];
                uint32_t w[3];
                chk_split2(x0, x1, w[0], w[1], w[2]);
                if (J < 3)
#pragma unroll
                    for (int p = 0; p < 3; ++p) xa[J < 3 ? J : 0][p][e] = w[p];
                if (is_w)
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(gW + (p * DK + at) * C + t) = w[p];      // W^T
            }
        }
    }
    pdl_trigger();
}

// The byte offset of 16-byte run `c` of row `r` in a tile of rows of RUNS runs: runs are swapped within their group of eight by the row's
// low bits, so that eight rows of one run lie in eight different banks' quads.
template <int RUNS>
__device__ __forceinline__ uint32_t dlc_at(int r, int c) { return (uint32_t)(r * RUNS + (c ^ (r & 7))) * 16; }

template <int DK>
__global__ void __launch_bounds__(CHK_THREADS, 1)
delta_chain_kernel(const __grid_constant__ DeltaArgs a) {
    constexpr int C = CHK_C, NT = CHK_THREADS, KH = DK / 2, KT = KH / 8, PART = C * DK * 2, BUF = 3 * PART;    // KH: keys a warp; bytes of a part, an operand
    extern __shared__ __align__(128) uint8_t dlc_bytes[];
    const uint32_t sW = chk_u32(dlc_bytes), sK = sW + 2 * BUF;       // W^T 3 x [DK][C], k 3 x [C][DK]; two buffers each
    float* sE = (float*)(dlc_bytes + 4 * BUF);               // [8 warps][C * 16]: halves of S^T W^T
    float* sD = sE + 8 * C * 16;                             // two of [DK]: a chunk's decays multiplied
    const int h = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lq = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    const int cols = warp & 3, k0 = (warp >> 2) * KH;        // this warp's 16 columns, its first key
    const int n_all = a.q_len[seq];
    if (n_all <= 0) return;
    const int dk = a.dk, dv = a.dv, dvp = a.tiles * DLC_COLS, n_chunks = (n_all + C - 1) / C, tile = blockIdx.z * (DLC_COLS / 16) + cols, v0 = tile * 16 + lg;
    // (the state before the wait, always: the rows' kernel triggers at its end, after a wait of its own, so everything before it is in memory)
    float* S_area = (float*)(a.state + (size_t)a.slot_ids[seq] * a.state_stride + a.state_offset) + (size_t)h * dk * dv;
    float S[KT][4];                                          // value columns v0 (+ 8), keys k0 + x * 8 + lq (+ 1)
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = k0 + x * 8 + lq + (e & 1), j = v0 + (e >> 1) * 8;
            S[x][e] = i < dk && j < dv ? S_area[(size_t)i * dv + j] : 0.f;
        }
    pdl_wait();
    const size_t block0 = delta_block(a, seq, 0, h), step = a.heads;
    auto ask = [&](int c) {                                  // chunk c's operands: W and the decays, then k
        const size_t blk = block0 + c * step;
        const uint8_t *w = (const uint8_t*)(a.wp + blk * (3 * C * DK)), *k = (const uint8_t*)(a.kp + blk * (3 * C * DK));
        const uint32_t to = (c & 1) * BUF;
#pragma unroll 4
        for (int idx = tid; idx < 3 * C * DK / 8; idx += NT) delta_cp16(sW + to + dlc_at<C / 8>(idx / (C / 8), idx % (C / 8)), w + idx * 16);
        if (tid < DK / 4) delta_cp16(chk_u32(sD + (c & 1) * DK + tid * 4), a.gc + blk * DK + tid * 4);
        delta_cp_commit();
#pragma unroll 4
        for (int idx = tid; idx < 3 * C * DK / 8; idx += NT) delta_cp16(sK + to + dlc_at<DK / 8>(idx / (DK / 8), idx % (DK / 8)), k + idx * 16);
        delta_cp_commit();
    };
    ask(0);
    for (int c = 0; c < n_chunks; ++c) {
        const size_t blk = block0 + c * step;
        if (c + 1 < n_chunks) ask(c + 1);                    // (its buffers were read before the last barrier)
        else { delta_cp_commit(); delta_cp_commit(); }
        const uint32_t w = sW + (c & 1) * BUF, k = sK + (c & 1) * BUF;
        float4* U = reinterpret_cast<float4*>(a.u + blk * (size_t)(C * dvp)) + (size_t)tile * (C * 4) + lane * 2;
        float u0[8][4];                                      // value columns v0 (+ 8), tokens x * 8 + lq (+ 1)
#pragma unroll
        for (int x = 0; x < 8; ++x) *reinterpret_cast<float4*>(u0[x]) = U[(x >> 1) * 64 + (x & 1)];
        // the state that this chunk starts from, for the outputs
        float4* sc = reinterpret_cast<float4*>(a.sc + blk * (size_t)(DK * dvp)) + (size_t)tile * (DK * 4) + k0 * 4 + lane * 2;
#pragma unroll
        for (int x = 0; x < KT; ++x) sc[(x >> 1) * 64 + (x & 1)] = make_float4(S[x][0], S[x][1], S[x][2], S[x][3]);
        delta_cp_wait<3>();
        __syncthreads();                                     // this chunk's W
        float u[8][2][4];                                    // this half of S^T W^T: the products of the first parts, and the small ones
#pragma unroll
        for (int x = 0; x < 8; ++x)
#pragma unroll
            for (int e = 0; e < 8; ++e) u[x][e >> 2][e & 3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KH / 16; ++ks) {
            uint32_t sa[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* s = S[2 * ks + (e >> 1)] + (e & 1) * 2;
                chk_split2(s[0], s[1], sa[0][e], sa[1][e], sa[2][e]);
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {           // 32 tokens at a time: four independent sums a product
                uint32_t wb[3][2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int pr = 0; pr < 2; ++pr)
                        chk_ldm4t(wb[p][pr], w + p * PART + dlc_at<C / 8>(k0 + ks * 16 + (lm & 1) * 8 + lr, (half * 2 + pr) * 2 + (lm >> 1)));
                CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const uint32_t* b = wb[pb][x >> 1] + (x & 1) * 2;
                        if (pa + pb == 0) chk_mma_sum<true>(u[half * 4 + x], sa[pa], b[0], b[1]);
                        else chk_mma_sum<false>(u[half * 4 + x], sa[pa], b[0], b[1]);
                    }
                }
            }
        }
        float4 *mine = (float4*)(sE + warp * (C * 16)) + lane, *other = (float4*)(sE + (warp ^ 4) * (C * 16)) + lane;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
#pragma unroll
            for (int e = 0; e < 4; ++e) u[x][0][e] += u[x][1][e];
            mine[x * 32] = make_float4(u[x][0][0], u[x][0][1], u[x][0][2], u[x][0][3]);
        }
        delta_cp_wait<2>();
        __syncthreads();                                     // the other half, and this chunk's k
        uint32_t ua[4][3][4];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const float4 y = other[x * 32];
            u0[x][0] -= u[x][0][0] + y.x;
            u0[x][1] -= u[x][0][1] + y.y;
            u0[x][2] -= u[x][0][2] + y.z;
            u0[x][3] -= u[x][0][3] + y.w;
#pragma unroll
            for (int f = 0; f < 2; ++f) chk_split2(u0[x][2 * f], u0[x][2 * f + 1], ua[x >> 1][0][(x & 1) * 2 + f], ua[x >> 1][1][(x & 1) * 2 + f], ua[x >> 1][2][(x & 1) * 2 + f]);
            if (k0 == 0) U[(x >> 1) * 64 + (x & 1)] = make_float4(u0[x][0], u0[x][1], u0[x][2], u0[x][3]);
        }
        const float* d = sD + (c & 1) * DK + k0;
#pragma unroll
        for (int x = 0; x < KT; ++x) {
            const float2 dd = *reinterpret_cast<const float2*>(d + x * 8 + lq);
            S[x][0] *= dd.x; S[x][1] *= dd.y; S[x][2] *= dd.x; S[x][3] *= dd.y;
        }
#pragma unroll
        for (int q = 0; q < KH / 32; ++q) {                  // 32 keys at a time
            float small[4][4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) small[x][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t kb[3][2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int pr = 0; pr < 2; ++pr)
                        chk_ldm4t(kb[p][pr], k + p * PART + dlc_at<DK / 8>(ks * 16 + (lm & 1) * 8 + lr, (k0 + q * 32) / 8 + pr * 2 + (lm >> 1)));
                CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const uint32_t* b = kb[pb][x >> 1] + (x & 1) * 2;
                        if (pa + pb == 0) chk_mma_sum<true>(S + q * 4 + x, ua[ks][pa], b[0], b[1]);
                        else chk_mma(small[x], ua[ks][pa], b[0], b[1]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[q * 4 + x][e] += small[x][e];
        }
        __syncthreads();                                     // W, k and the halves have been read
    }
    pdl_trigger();
    delta_cp_wait<0>();
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = k0 + x * 8 + lq + (e & 1), j = v0 + (e >> 1) * 8;
            if (i < dk && j < dv) S_area[(size_t)i * dv + j] = S[x][e];
        }
}

template <int DK, int NB>
__global__ void __launch_bounds__(CHK_THREADS, 2)
delta_outputs_kernel(const __grid_constant__ DeltaArgs a) {
    constexpr int C = CHK_C;
    extern __shared__ __align__(128) uint8_t dlc_bytes[];
    pdl_trigger();
    const int dvp = a.tiles * DLC_COLS, spans = dvp / NB, lane = threadIdx.x & 31;
    const int h = blockIdx.x, seq = blockIdx.y, c = blockIdx.z / spans, col0 = (blockIdx.z - c * spans) * NB;
    const int n = min(C, a.q_len[seq] - c * C), r0 = a.q_start[seq] + c * C;
    if (n <= 0) return;
    const size_t block = delta_block(a, seq, c, h);
    const bool pairs = (a.dv & 1) == 0 && (a.out_stride & 1) == 0 && ((uintptr_t)a.out & 7) == 0;
    const size_t tile = (col0 + chk_out_col<NB>()) / 16;
    const float4 *sc = reinterpret_cast<const float4*>(a.sc + block * (size_t)(DK * dvp)) + tile * (DK * 4) + lane * 2;
    const float4 *U = reinterpret_cast<const float4*>(a.u + block * (size_t)(C * dvp)) + tile * (C * 4) + lane * 2;
    pdl_wait();
    chk_outputs<DK, 3, NB, false>(
        dlc_bytes, a.qd + block * (C * DK), a.p + block * (C * C), false,
        [&](float* x, int ks) {
            const float4 v = sc[ks * 64], w = sc[ks * 64 + 1];
            x[0] = v.x; x[1] = v.y; x[2] = w.x; x[3] = w.y;
            x[4] = v.z; x[5] = v.w; x[6] = w.z; x[7] = w.w;
        },
        [](__nv_bfloat16*) {},
        [&](uint32_t (*b)[4], int ks, const __nv_bfloat16*) {
            const float4 v = U[ks * 64], w = U[ks * 64 + 1];
            chk_split2(v.x, v.y, b[0][0], b[1][0], b[2][0]);
            chk_split2(w.x, w.y, b[0][1], b[1][1], b[2][1]);
            chk_split2(v.z, v.w, b[0][2], b[1][2], b[2][2]);
            chk_split2(w.z, w.w, b[0][3], b[1][3], b[2][3]);
        },
        [&](int t, int at, float x, float y) {
            const int col = col0 + at;
            if (t >= n) return;
            float* to = a.out + (size_t)(r0 + t) * a.out_stride + (size_t)h * a.dv + col;
            if (pairs && col < a.dv) *reinterpret_cast<float2*>(to) = make_float2(x, y);
            else {
                if (col < a.dv) to[0] = x;
                if (col + 1 < a.dv) to[1] = y;
            }
        });
}

long long dlc_floats(long long blocks, int dk, int dv) {
    const long long dkp = dk <= 64 ? 64 : 128, dvp = (dv + DLC_COLS - 1) / DLC_COLS * DLC_COLS;
    // W and k in parts, decayed q, U, P, the decays, the states
    return blocks * (2 * 3 * CHK_C * dkp / 2 + CHK_C * dkp + CHK_C * dvp + CHK_C * CHK_C + dkp + dkp * dvp);
}

template <typename T, int DK>
static int launch_dlc(DeltaArgs a, int n_seqs, long long blocks, float* work, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(delta_rows_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, dlc_rows_smem<DK>());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chain_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, dlc_chain_smem<DK>());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_outputs_kernel<DK, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (chk_out_smem<DK, 0>()));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_outputs_kernel<DK, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (chk_out_smem<DK, 0>()));
        if (e != cudaSuccess) { braid_set_error("delta_rule: cannot reserve shared memory: %s", cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    a.tiles = (a.dv + DLC_COLS - 1) / DLC_COLS;
    const long long dvp = (long long)a.tiles * DLC_COLS;
    a.qd = work;
    a.u = a.qd + blocks * CHK_C * DK;
    a.p = a.u + blocks * CHK_C * dvp;
    a.sc = a.p + blocks * CHK_C * CHK_C;
    a.gc = a.sc + blocks * DK * dvp;
    a.wp = (__nv_bfloat16*)(a.gc + blocks * DK);
    a.kp = a.wp + blocks * 3 * CHK_C * DK;
    braid_launch(delta_rows_kernel<T, DK>, dim3(a.heads, n_seqs, a.max_chunks), dim3(CHK_THREADS), (size_t)dlc_rows_smem<DK>(), s, a);
    braid_launch(delta_chain_kernel<DK>, dim3(a.heads, n_seqs, a.tiles), dim3(CHK_THREADS), (size_t)dlc_chain_smem<DK>(), s, a);
    const size_t smem = chk_out_smem<DK, 0>();
    if (a.tiles % 2) braid_launch(delta_outputs_kernel<DK, 64>, dim3(a.heads, n_seqs, a.max_chunks * a.tiles), dim3(CHK_THREADS), smem, s, a);
    else braid_launch(delta_outputs_kernel<DK, 128>, dim3(a.heads, n_seqs, a.max_chunks * (a.tiles / 2)), dim3(CHK_THREADS), smem, s, a);
    BRAID_LAUNCH_CHECK();
}

int dlc_launch(const DeltaArgs& a, int dtype, int n_seqs, long long blocks, float* work, cudaStream_t s) {
    if (dtype == BRAID_F32) return a.dk <= 64 ? launch_dlc<float, 64>(a, n_seqs, blocks, work, s) : launch_dlc<float, 128>(a, n_seqs, blocks, work, s);
    return a.dk <= 64 ? launch_dlc<__nv_bfloat16, 64>(a, n_seqs, blocks, work, s) : launch_dlc<__nv_bfloat16, 128>(a, n_seqs, blocks, work, s);
}
