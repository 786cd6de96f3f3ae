// The linear recurrence with one decay a head (state-space duality) over chunks of a prompt, on the tensor cores, for bfloat16 rows:
//   S <- a_t S + (dt_t k_t) v_t^T,   o_t = S^T (q_scale q_t) + skip v_t,   S [dk, 64 value columns] float32
// with dt = softplus(d + bias), a = exp(-exp(A_log) dt) (scan.cu's DECAY_HEAD).  With D(s, t) the product of the decays after s up to t,
// D(0, t) from the chunk's start, and S_0 the state a chunk of 64 tokens starts from:
//   P_ts = (q_t . k_s) dt_s D(s, t)  (s <= t)        O = diag(D(0, t)) Q S_0 + P V
//   S_64 = D(0, 64) S_0 + K^T (dt_t D(t, 64) v_t)
//
// q, k and v are bfloat16 numbers, so their products are exact in the tensor cores.  What is float32 (S_0, P, the weighted values)
// goes in as the sum of three bfloat16 numbers, 24 bits, in three products that add into one float32 accumulator: nothing is
// rounded to fewer bits than the walk token by token keeps, only the order of the sums differs (the tests hold the error beside
// float64 to the walk's own).  The decays are products of decays, never
// differences of logarithms.  A token's numbers never reach the tokens before it, be they infinite: the block on the diagonal
// selects the later tokens away instead of multiplying them by zero.
//
// A CTA of four warps owns (head, sequence, 64 value columns) and walks the sequence's chunks.  A warp owns 16 value columns and keeps their
// transposed state in its accumulators, which are the operand of S^T Q^T as they are: the state never passes through shared memory.
// P is worked out by rows of 16 tokens a warp and shared as three parts.  The next chunk is on its way while one is worked on (two
// buffers); two CTAs an SM (112 KB of shared memory at dk 128).  Bound by mma.sync: some 500 a warp and chunk at 11 to 16 cycles each with one
// warp a scheduler, 12,300 cycles a chunk with the splits between them.  us beside the form before, whose state went to shared memory in
// parts for every chunk, / the walk token by token in two passes over chunks (scan.cu), heads of 128 x 64: 64 heads, 2,048 tokens
// 256 / 262 / 478, 1,500 + 1,200 + 900 tokens 219 / 232 / 842, 64 tokens 16.5 / 22 / 31; 128 heads, 2,048 tokens 268 / 267 / 929.  32 heads of
// 64 x 64: 3 sequences 135 / 156 / 244, 300 tokens 33 / 38 / 68.  A long prompt on few CTAs is a
// chain that leaves the machine idle (8 heads of 128 x 64, 2,048 tokens: 243 us beside 130): such steps stay with
// the walk whose chunks run side by side, by `ssd_pays` (api.py), which holds both forms' times.
#include "chunk_mma.cuh"

#define SSD_C 64
#define SSD_P 64
#define SSD_THREADS 128

struct SsdArgs {
    const __nv_bfloat16 *q, *k, *v, *gate, *gate_bias, *a_log, *skip;
    long long q_stride, k_stride, v_stride, gate_stride;
    float* out; long long out_stride;
    uint8_t* state; long long state_stride, state_offset;
    const int *q_start, *q_len, *slot_ids;
    int heads, groups, dv;
    float q_scale;
    int settled;                 // the state may be read before the wait (common.cuh)
};

// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void ssd_copy16(uint32_t dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// two bfloat16 numbers, those that are not finite replaced by zero
__device__ __forceinline__ uint32_t ssd_finite(uint32_t w) {
    return ((w & 0x7f80u) == 0x7f80u ? 0u : w & 0xffffu) | ((w & 0x7f800000u) == 0x7f800000u ? 0u : w & 0xffff0000u);
}
// The byte offset of 16-byte run `c` of row `r` in a tile of rows of RUNS runs (8 or 16): runs are swapped within their group of eight
// by the row's low bits, so that eight rows of one run lie in eight different banks' quads.
template <int RUNS>
__device__ __forceinline__ uint32_t ssd_at(int r, int c) { return (uint32_t)(r * RUNS + (c ^ (r & 7))) * 16; }

// A token's numbers of the chunk
struct SsdToken {
    float head;                  // its decay and those before it in its block of 16, multiplied
    float tail;                  // those after it in its block, times its step
    float start;                 // D(0, t) q_scale
    float end;                   // dt_t D(t, 64)
};
template <int DK> constexpr int ssd_smem() {
    return 2 * (2 * SSD_C * DK * 2 + SSD_C * SSD_P * 2) + 3 * SSD_C * SSD_C * 2 + SSD_C * 17 * 4 + SSD_C * 16 + 8 * 4;
}

template <int DK>
__global__ void __launch_bounds__(SSD_THREADS, 2)
ssd_chunk_kernel(const __grid_constant__ SsdArgs a) {
    constexpr int C = SSD_C, P = SSD_P, QR = DK / 8, KT = DK / 8, QB = C * DK * 2, VB = C * P * 2, PB = C * C * 2;
    extern __shared__ __align__(128) uint8_t ssd_sm[];
    const uint32_t sQ = chk_u32(ssd_sm), sK = sQ + 2 * QB, sV = sK + 2 * QB, sP = sV + 2 * VB;      // q, k, v: two buffers; P: three parts
    float* sD = (float*)(ssd_sm + 4 * QB + 2 * VB + 3 * PB);     // [t][17]: dt_s D(s, t), s in t's block of 16
    SsdToken* tok = (SsdToken*)(sD + C * 17);                // [C]
    float* s_block = (float*)(tok + C);                      // [4]: a block's decays multiplied
    int* s_odd = (int*)(s_block + 4);                        // [4]: values that are not finite
    pdl_trigger();
    const int h = blockIdx.x, seq = blockIdx.y, j0 = blockIdx.z * P, tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q2 = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    const int n = a.q_len[seq], r0 = a.q_start[seq];
    if (n <= 0) return;
    const int grp = h / (a.heads / a.groups), cw = warp * 16;
    const float head_a = -expf(to_f32(a.a_log[h])), head_bias = to_f32(a.gate_bias[h]), skip = a.skip ? to_f32(a.skip[h]) : 0.f;
    float* S_area = (float*)(a.state + (size_t)a.slot_ids[seq] * a.state_stride + a.state_offset) + (size_t)h * DK * a.dv + j0 + cw + g;
    if (!a.settled) pdl_wait();
    float S[KT][4];                                          // S^T: value columns cw + g (+ 8), keys x * 8 + q2 (+ 1)
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[x][e] = S_area[(size_t)(x * 8 + q2 + (e & 1)) * a.dv + (e >> 1) * 8];
    pdl_wait();
    auto ask = [&](int t0, int buf) {                        // the tokens from t0 on, zeros past the sequence
        const int nt = min(C, n - t0);
#pragma unroll 4
        for (int i = tid; i < C * QR; i += SSD_THREADS) {
            const int r = i / QR, c = i % QR;
            const bool in = r < nt;
            const size_t row = (size_t)(r0 + t0 + (in ? r : 0));
            ssd_copy16(sQ + buf * QB + ssd_at<QR>(r, c), a.q + row * a.q_stride + (size_t)grp * DK + c * 8, in);
            ssd_copy16(sK + buf * QB + ssd_at<QR>(r, c), a.k + row * a.k_stride + (size_t)grp * DK + c * 8, in);
        }
#pragma unroll
        for (int i = tid; i < C * 8; i += SSD_THREADS) {
            const int r = i / 8, c = i % 8;
            const bool in = r < nt;
            ssd_copy16(sV + buf * VB + ssd_at<8>(r, c), a.v + (size_t)(r0 + t0 + (in ? r : 0)) * a.v_stride + (size_t)h * a.dv + j0 + c * 8, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto gate_of = [&](int t) { return tid < C && t < n ? to_f32(a.gate[(size_t)(r0 + t) * a.gate_stride + h]) : 0.f; };
    ask(0, 0);
    float z = gate_of(tid);
    for (int t0 = 0, buf = 0; t0 < n; t0 += C, buf ^= 1) {
        const int nt = min(C, n - t0);
        const uint32_t q = sQ + buf * QB, k = sK + buf * QB, v = sV + buf * VB;
        const uint8_t* v_bytes = ssd_sm + 4 * QB + buf * VB;
        if (tid < C) {                                       // a thread a token; past the end: no decay, no step
            float dt = 0.f, dec = 1.f;
            if (tid < nt) {
                const float x = z + head_bias;
                dt = x > 20.f ? x : log1pf(expf(x));
                dec = expf(head_a * dt);
            }
            const int l = lane & 15;
            float run = dt, pre = dec, suf = dec;
            sD[tid * 17 + l] = run;
#pragma unroll
            for (int r = 1; r < 16; ++r) {                   // down the tokens of the block
                const float d = __shfl_down_sync(0xffffffffu, dec, r, 16);
                if (l + r < 16) {
                    run *= d;
                    sD[(tid + r) * 17 + l] = run;
                }
            }
#pragma unroll
            for (int r = 1; r < 16; r <<= 1) {
                const float x = __shfl_up_sync(0xffffffffu, pre, r, 16), y = __shfl_down_sync(0xffffffffu, suf, r, 16);
                if (l >= r) pre *= x;
                if (l + r < 16) suf *= y;
            }
            const float after = __shfl_down_sync(0xffffffffu, suf, 1, 16);
            tok[tid].head = pre;
            tok[tid].tail = l < 15 ? dt * after : dt;
            if (l == 15) s_block[tid >> 4] = pre;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                     // the chunk is there; the one before has been read
        if (t0 + C < n) {
            ask(t0 + C, buf ^ 1);
            z = gate_of(t0 + C + tid);
        }
        const float b0 = s_block[0], b1 = s_block[1], b2 = s_block[2], b3 = s_block[3], all = b0 * b1 * b2 * b3;
        if (tid < C) {
            const int b = tid >> 4;
            tok[tid].start = tok[tid].head * (b == 0 ? 1.f : b == 1 ? b0 : b == 2 ? b0 * b1 : b0 * b1 * b2) * a.q_scale;
            tok[tid].end = tok[tid].tail * (b == 3 ? 1.f : b == 2 ? b3 : b == 1 ? b2 * b3 : b1 * b2 * b3);
        } else if (warp == 3) {                              // which blocks of 16 tokens hold values that are not finite
#pragma unroll
            for (int b = 0; b < C / 16; ++b) {
                uint32_t top = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 u = *reinterpret_cast<const uint4*>(v_bytes + (b * 128 + i * 32 + lane) * 16);
                    top |= ((u.x & 0x7f807f80u) + 0x00800080u) | ((u.y & 0x7f807f80u) + 0x00800080u) |
                           ((u.z & 0x7f807f80u) + 0x00800080u) | ((u.w & 0x7f807f80u) + 0x00800080u);
                }
                const bool any = __any_sync(0xffffffffu, top & 0x80008000u);
                if (lane == 0) s_odd[b] = any;
            }
        }
        {                                                    // P: the warp's 16 tokens against the tokens up to them
            float qk[8][4];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) qk[x][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < DK / 16; ++ks) {
                uint32_t qa[4];
                chk_ldm4(qa, q + ssd_at<QR>(cw + (lm & 1) * 8 + lr, ks * 2 + (lm >> 1)));
#pragma unroll
                for (int pr = 0; pr < 4; ++pr)
                    if (pr <= warp) {
                        uint32_t kb[4];
                        chk_ldm4(kb, k + ssd_at<QR>(pr * 16 + (lm >> 1) * 8 + lr, ks * 2 + (lm & 1)));
                        chk_mma(qk[2 * pr], qa, kb[0], kb[1]);
                        chk_mma(qk[2 * pr + 1], qa, kb[2], kb[3]);
                    }
            }
            const float h0 = tok[cw + g].head * a.q_scale, h1 = tok[cw + g + 8].head * a.q_scale;
            float between = 1.f;
#pragma unroll
            for (int pr = 3; pr >= 0; --pr) {                // blocks of tokens s, from the warp's own back
                if (pr > warp) continue;
                if (pr < warp - 1) between *= pr == 0 ? b1 : b2;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int s = half * 8 + q2;
                    float* x = qk[2 * pr + half];
                    if (pr == warp) {                        // tokens after this one are left out, whatever their products are
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int t = g + (e >> 1) * 8;
                            x[e] = s + (e & 1) <= t ? x[e] * (sD[(cw + t) * 17 + s + (e & 1)] * a.q_scale) : 0.f;
                        }
                    } else {
                        const float f0 = tok[pr * 16 + s].tail * between, f1 = tok[pr * 16 + s + 1].tail * between;
                        x[0] *= f0 * h0; x[1] *= f1 * h0; x[2] *= f0 * h1; x[3] *= f1 * h1;
                    }
                    uint32_t lo[3], hi[3];
                    chk_split2(x[0], x[1], lo[0], lo[1], lo[2]);
                    chk_split2(x[2], x[3], hi[0], hi[1], hi[2]);
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sP + p * PB + ssd_at<8>(cw + g, pr * 2 + half) + q2 * 2), "r"(lo[p]) : "memory");
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sP + p * PB + ssd_at<8>(cw + g + 8, pr * 2 + half) + q2 * 2), "r"(hi[p]) : "memory");
                    }
                }
            }
        }
        float o[8][2][4];                                    // O^T, value columns cw + g (+ 8), tokens x * 8 + q2 (+ 1)
#pragma unroll
        for (int x = 0; x < 8; ++x)
#pragma unroll
            for (int e = 0; e < 8; ++e) o[x][e >> 2][e & 3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < DK / 16; ++ks) {               // S^T Q^T
            uint32_t sa[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* s = S[2 * ks + (e >> 1)] + (e & 1) * 2;
                chk_split2(s[0], s[1], sa[0][e], sa[1][e], sa[2][e]);
            }
            uint32_t qb[4][4];
#pragma unroll
            for (int pr = 0; pr < 4; ++pr) chk_ldm4(qb[pr], q + ssd_at<QR>(pr * 16 + (lm >> 1) * 8 + lr, ks * 2 + (lm & 1)));
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const uint32_t* b = qb[x >> 1] + (x & 1) * 2;
                    if (p == 0) chk_mma_sum<true>(o[x], sa[p], b[0], b[1]);
                    else chk_mma_sum<false>(o[x], sa[p], b[0], b[1]);
                }
        }
        __syncthreads();                                     // P and the tokens' numbers are there
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const float d0 = tok[x * 8 + q2].start, d1 = tok[x * 8 + q2 + 1].start;
#pragma unroll
            for (int w = 0; w < 2; ++w) { o[x][w][0] *= d0; o[x][w][1] *= d1; o[x][w][2] *= d0; o[x][w][3] *= d1; }
        }
        uint32_t wv[4][3][4];                                // (dt_t D(t, 64) v_t)^T in parts, for the state
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {                     // V^T P^T, 16 tokens s at a time
            uint32_t va[4];
            chk_ldm4t(va, v + ssd_at<8>(ks * 16 + (lm >> 1) * 8 + lr, cw / 8 + (lm & 1)));
            const bool odd = s_odd[ks];
#pragma unroll
            for (int pr = 0; pr < 4; ++pr) {
                if (pr < ks) continue;
                uint32_t pb[3][4], vf[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) vf[e] = odd && pr == ks ? ssd_finite(va[e]) : va[e];
#pragma unroll
                for (int p = 0; p < 3; ++p) chk_ldm4(pb[p], sP + p * PB + ssd_at<8>(pr * 16 + (lm >> 1) * 8 + lr, ks * 2 + (lm & 1)));
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (p == 0) chk_mma_sum<true>(o[2 * pr + x], vf, pb[p][2 * x], pb[p][2 * x + 1]);
                        else chk_mma_sum<false>(o[2 * pr + x], vf, pb[p][2 * x], pb[p][2 * x + 1]);
                    }
            }
            if (odd) {                                       // the values left out on the diagonal, for their own and later tokens alone
#pragma unroll 1
                for (int s = 0; s < 16; ++s)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int row = ks * 16 + s, col = cw + g + e * 8;
                        const float y = to_f32(*reinterpret_cast<const __nv_bfloat16*>(v_bytes + ssd_at<8>(row, col >> 3) + (col & 7) * 2));
                        if (isfinite(y)) continue;
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            const int t = (x >> 1) * 8 + q2 + (x & 1);
                            if (s > t) continue;
                            float w = 0.f;
#pragma unroll
                            for (int p = 0; p < 3; ++p)
                                w += to_f32(*reinterpret_cast<const __nv_bfloat16*>(ssd_sm + 4 * QB + 2 * VB + p * PB + ssd_at<8>(ks * 16 + t, row >> 3) + (row & 7) * 2));
                            float* sum = &o[2 * ks + (x >> 1)][0][e * 2 + (x & 1)];
                            *sum = fmaf(w, y, *sum);
                        }
                    }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {                    // va[e]: column cw + g + (e & 1) * 8, tokens ks * 16 + (e >> 1) * 8 + q2 and the next
                const int t = ks * 16 + (e >> 1) * 8 + q2;
                const float v0 = __uint_as_float(va[e] << 16), v1 = __uint_as_float(va[e] & 0xffff0000u);
                float* y = o[2 * ks + (e >> 1)][0] + (e & 1) * 2;
                if (a.skip) {
                    y[0] = fmaf(skip, v0, y[0]);
                    y[1] = fmaf(skip, v1, y[1]);
                }
                chk_split2(v0 * tok[t].end, v1 * tok[t + 1].end, wv[ks][0][e], wv[ks][1][e], wv[ks][2][e]);
            }
        }
#pragma unroll
        for (int x = 0; x < 8; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = x * 8 + q2 + (e & 1);
                if (t < nt) a.out[(size_t)(r0 + t0 + t) * a.out_stride + (size_t)h * a.dv + j0 + cw + g + (e >> 1) * 8] = o[x][0][e] + o[x][1][e];
            }
#pragma unroll
        for (int x = 0; x < KT; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[x][e] *= all;
#pragma unroll
        for (int part = 0; part < DK / 32; ++part) {         // the state, 32 keys at a time
            float small[4][4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) small[x][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t kb[2][4];
#pragma unroll
                for (int pr = 0; pr < 2; ++pr) chk_ldm4t(kb[pr], k + ssd_at<QR>(ks * 16 + (lm & 1) * 8 + lr, part * 4 + pr * 2 + (lm >> 1)));
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const uint32_t* b = kb[x >> 1] + (x & 1) * 2;
                        if (p == 0) chk_mma_sum<true>(S + part * 4 + x, wv[ks][p], b[0], b[1]);
                        else chk_mma(small[x], wv[ks][p], b[0], b[1]);
                    }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[part * 4 + x][e] += small[x][e];
        }
    }
#pragma unroll
    for (int x = 0; x < KT; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) S_area[(size_t)(x * 8 + q2 + (e & 1)) * a.dv + (e >> 1) * 8] = S[x][e];
}

template <int DK>
static int launch_ssd(const SsdArgs& a, int n_seqs, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(ssd_chunk_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, ssd_smem<DK>());
        if (e != cudaSuccess) { braid_set_error("ssd_scan: cannot reserve %d bytes of shared memory: %s", ssd_smem<DK>(), cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    braid_launch(ssd_chunk_kernel<DK>, dim3(a.heads, n_seqs, a.dv / SSD_P), dim3(SSD_THREADS), (size_t)ssd_smem<DK>(), s, a);
    BRAID_LAUNCH_CHECK();
}

// bfloat16 rows and gates; dk 64 or 128, dv a multiple of 64, rows of q, k and v on 16 bytes.
extern "C" int braid_ssd_scan(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                              const void* gate, long long gate_stride, const void* gate_bias, const void* a_log, const void* skip,
                              float* out, long long out_stride, void* state, long long state_stride, long long state_offset,
                              const int* q_start, const int* q_len, const int* slot_ids, int n_seqs, int heads, int groups, int dk, int dv,
                              float q_scale, int settled, void* stream) {
    if (n_seqs <= 0) return BRAID_OK;
    if (heads <= 0 || groups <= 0 || heads % groups) BRAID_REFUSE("ssd_scan: %d heads do not divide into %d groups", heads, groups);
    if ((dk != 64 && dk != 128) || dv <= 0 || dv % SSD_P) BRAID_REFUSE("ssd_scan: built for keys of 64 or 128 and values in multiples of 64, not %d x %d", dk, dv);
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) || q_stride % 8 || k_stride % 8 || v_stride % 8) BRAID_REFUSE("ssd_scan: rows must start on 16 bytes");
    if (((uintptr_t)out & 7) || out_stride % 2 || !state || (((uintptr_t)state | (uintptr_t)state_offset | (uintptr_t)state_stride) & 7)) BRAID_REFUSE("ssd_scan: results and state must start on 8 bytes");
    if (!gate_bias || !a_log || n_seqs > 65535 || dv / SSD_P > 65535) BRAID_REFUSE("ssd_scan: a bias and A_log are required, and the step must fit a launch");
    using B = const __nv_bfloat16*;
    SsdArgs a{(B)q, (B)k, (B)v, (B)gate, (B)gate_bias, (B)a_log, (B)skip, q_stride, k_stride, v_stride, gate_stride, out, out_stride,
              (uint8_t*)state, state_stride, state_offset, q_start, q_len, slot_ids, heads, groups, dv, q_scale, settled};
    return dk == 64 ? launch_ssd<64>(a, n_seqs, (cudaStream_t)stream) : launch_ssd<128>(a, n_seqs, (cudaStream_t)stream);
}
