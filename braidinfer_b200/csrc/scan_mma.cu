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
// A CTA of four warps owns (head, sequence, 64 value columns) and walks the sequence's chunks, the state in its accumulator
// registers (a warp a quarter of the key rows); a warp owns 16 tokens of a chunk's output, and its P goes from the accumulators of
// Q K^T straight into the operands of P V.  Two CTAs an SM (108 KB of shared memory at dk 128).  The walk token by token in two
// passes over chunks (scan.cu) is bound by shared-memory reads and shuffles.  Measured beside it, us, heads of 128 x 64:
// 64 heads, 2,048 tokens 262 beside 478, 1,500 + 1,200 + 900 tokens 232 / 842, 8 x 64 tokens 36 / 97, 4 x 24 tokens 22 / 35; 128 heads,
// 2,048 tokens 267 / 929.  32 heads of 64 x 64: 3 sequences 156 / 244, 300 tokens 38 / 68.  A long prompt on few CTAs is a
// chain that leaves the machine idle (8 us a chunk; 8 heads of 128 x 64, 2,048 tokens: 259 us beside 129): such steps stay with
// the walk whose chunks run side by side, by `ssd_pays` (api.py), which holds both forms' times.
#include "common.cuh"
#include <type_traits>

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
};

__device__ __forceinline__ uint32_t ssd_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ssd_ldm4(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ssd_ldm4t(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ssd_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void ssd_copy16(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ssd_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// x = the sum of three bfloat16 numbers to float32's 24 bits; two x at once, packed.  The first two saturate, so that a number past the
// largest bfloat16 one is still a sum of finite parts; an infinity is left over for the third.
__device__ __forceinline__ void ssd_split2(float x0, float x1, uint32_t* w) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i < 2) {
            asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w[i]) : "f"(x1), "f"(x0));
        } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        x0 -= __uint_as_float(w[i] << 16);
        x1 -= __uint_as_float(w[i] & 0xffff0000u);
    }
}
// two bfloat16 numbers, those that are not finite replaced by zero
__device__ __forceinline__ uint32_t ssd_finite(uint32_t w) {
    return ((w & 0x7f80u) == 0x7f80u ? 0u : w & 0xffffu) | ((w & 0x7f800000u) == 0x7f800000u ? 0u : w & 0xffff0000u);
}
// The byte offset of 16-byte run `c` of row `r` in a tile of rows of RUNS runs (8 or 16): runs are swapped within their group of eight
// by the row's low bits, so that eight rows of one run lie in eight different banks' quads.
template <int RUNS>
__device__ __forceinline__ uint32_t ssd_at(int r, int c) { return (uint32_t)(r * RUNS + (c ^ (r & 7))) * 16; }

template <int DK> constexpr int ssd_smem() {
    return SSD_C * DK * 2 * 2 + SSD_C * SSD_P * 2 + SSD_C * (SSD_C + 1) * 4 + 3 * DK * SSD_P * 2 + 4 * SSD_C * 4 + SSD_C / 16 * 4;
}

template <int DK>
__global__ void __launch_bounds__(SSD_THREADS, 2)
ssd_chunk_kernel(SsdArgs a) {
    constexpr int C = SSD_C, P = SSD_P, QR = DK / 8, MT = DK / 64;      // MT: 16-row tiles of the state a warp
    extern __shared__ __align__(16) uint8_t ssd_sm[];
    uint8_t* sQ = ssd_sm;                                    // [C][DK] bf16; from the state update on, with sD: the weighted values, 3 x [C][P]
    uint8_t* sD_ = sQ + C * DK * 2;
    float* sD = (float*)sD_;                                 // [t][s], rows of C + 1: dt_s D(s, t)
    uint8_t* sK = sD_ + C * (C + 1) * 4;                     // [C][DK]
    uint8_t* sV = sK + C * DK * 2;                           // [C][P]
    uint8_t* sS = sV + C * P * 2;                            // 3 x [DK][P]: the state the chunk starts from
    float* s_a = (float*)(sS + 3 * DK * P * 2);              // decays
    float* s_dt = s_a + C;
    float* s_d0 = s_dt + C;                                  // D(0, t)
    float* s_w = s_d0 + C;                                   // dt_t D(t, 64)
    int* s_odd = (int*)(s_w + C);                            // [C / 16]
    uint8_t* sW = sQ;
    static_assert(3 * C * P * 2 <= C * DK * 2 + C * (C + 1) * 4, "the weighted values fit where q and the decays were");
    pdl_trigger();
    const int h = blockIdx.x, seq = blockIdx.y, j0 = blockIdx.z * P, tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q2 = (lane & 3) * 2;
    const int n = a.q_len[seq], r0 = a.q_start[seq];
    if (n <= 0) return;
    const int grp = h / (a.heads / a.groups);
    const float head_a = -expf(to_f32(a.a_log[h])), head_bias = to_f32(a.gate_bias[h]), skip = a.skip ? to_f32(a.skip[h]) : 0.f;
    float* S_area = (float*)(a.state + (size_t)a.slot_ids[seq] * a.state_stride + a.state_offset) + (size_t)h * DK * a.dv + j0;
    pdl_wait();
    const int i0 = warp * (DK / 4);                          // this warp's rows of the state
    float S[MT][8][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 v = *reinterpret_cast<const float2*>(S_area + (size_t)(i0 + m * 16 + g + e * 8) * a.dv + t * 8 + q2);
                S[m][t][2 * e] = v.x;
                S[m][t][2 * e + 1] = v.y;
            }
    for (int t0 = 0; t0 < n; t0 += C) {
        const int nt = min(C, n - t0);
        // everything of the chunk asked for at once; it arrives under the split of the state
#pragma unroll
        for (int i = tid; i < C * QR; i += SSD_THREADS) {
            const int r = i / QR, c = i % QR;
            const bool in = r < nt;
            const size_t row = (size_t)(r0 + t0 + (in ? r : 0));
            ssd_copy16(sQ + ssd_at<QR>(r, c), a.q + row * a.q_stride + (size_t)grp * DK + c * 8, in);
            ssd_copy16(sK + ssd_at<QR>(r, c), a.k + row * a.k_stride + (size_t)grp * DK + c * 8, in);
        }
#pragma unroll
        for (int i = tid; i < C * 8; i += SSD_THREADS) {
            const int r = i / 8, c = i % 8;
            const bool in = r < nt;
            ssd_copy16(sV + ssd_at<8>(r, c), a.v + (size_t)(r0 + t0 + (in ? r : 0)) * a.v_stride + (size_t)h * a.dv + j0 + c * 8, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (tid < C) {                                       // tokens past the end: no decay, no step
            float dt = 0.f, dec = 1.f;
            if (tid < nt) {
                const float x = to_f32(a.gate[(size_t)(r0 + t0 + tid) * a.gate_stride + h]) + head_bias;
                dt = x > 20.f ? x : log1pf(expf(x));
                dec = expf(head_a * dt);
            }
            s_dt[tid] = dt;
            s_a[tid] = dec;
        }
        // the state in three parts
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < 8; ++t)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    uint32_t w[3];
                    ssd_split2(S[m][t][2 * e], S[m][t][2 * e + 1], w);
                    const int r = i0 + m * 16 + g + e * 8;
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(sS + p * DK * P * 2 + ssd_at<8>(r, t) + q2 * 2) = w[p];
                }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (tid < C) {                                       // a thread a column s: products down the tokens
            float run = s_dt[tid];
#pragma unroll 8
            for (int t = 0; t < C; ++t) {
                if (t > tid) run *= s_a[t];
                sD[t * (C + 1) + tid] = t < tid ? 0.f : run;
            }
            s_w[tid] = run;
        } else if (tid == C) {
            float run = 1.f;
#pragma unroll 8
            for (int t = 0; t < C; ++t) {
                run *= s_a[t];
                s_d0[t] = run;
            }
        } else if (warp == 3) {                              // meanwhile: which blocks of 16 tokens hold values that are not finite
#pragma unroll
            for (int b = 0; b < C / 16; ++b) {
                uint32_t top = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 u = *reinterpret_cast<const uint4*>(sV + (b * 128 + i * 32 + lane) * 16);
                    top |= ((u.x & 0x7f807f80u) + 0x00800080u) | ((u.y & 0x7f807f80u) + 0x00800080u) |
                           ((u.z & 0x7f807f80u) + 0x00800080u) | ((u.w & 0x7f807f80u) + 0x00800080u);
                }
                const bool any = __any_sync(0xffffffffu, top & 0x80008000u);
                if (lane == 0) s_odd[b] = any;
            }
        }
        // Q K^T, the warp's 16 tokens against the tokens up to them
        const int tw = warp * 16;
        float o[8][4], qk[8][4];
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) { o[t][e] = 0.f; qk[t][e] = 0.f; }
        const int lr = lane & 7, lm = lane >> 3;             // row and matrix of this lane's address in an ldmatrix of four
#pragma unroll
        for (int ks = 0; ks < DK / 16; ++ks) {
            uint32_t qa[4];
            ssd_ldm4(qa, ssd_u32(sQ) + ssd_at<QR>(tw + (lm & 1) * 8 + lr, ks * 2 + (lm >> 1)));
#pragma unroll
            for (int pr = 0; pr < 4; ++pr)                   // 16 tokens s at a time
                if (pr <= warp) {
                    uint32_t kb[4];
                    ssd_ldm4(kb, ssd_u32(sK) + ssd_at<QR>(pr * 16 + (lm >> 1) * 8 + lr, ks * 2 + (lm & 1)));
                    ssd_mma(qk[2 * pr], qa, kb[0], kb[1]);
                    ssd_mma(qk[2 * pr + 1], qa, kb[2], kb[3]);
                }
            // and Q S_0: the state's key rows ks * 16 ...
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int pr = 0; pr < 4; ++pr) {
                    uint32_t sb[4];
                    ssd_ldm4t(sb, ssd_u32(sS) + p * DK * P * 2 + ssd_at<8>(ks * 16 + (lm & 1) * 8 + lr, pr * 2 + (lm >> 1)));
                    ssd_mma(o[2 * pr], qa, sb[0], sb[1]);
                    ssd_mma(o[2 * pr + 1], qa, sb[2], sb[3]);
                }
        }
        __syncthreads();                                     // the decays are there
        const float d0 = s_d0[tw + g], d1 = s_d0[tw + g + 8];
#pragma unroll
        for (int t = 0; t < 8; ++t) { o[t][0] *= d0; o[t][1] *= d0; o[t][2] *= d1; o[t][3] *= d1; }
        // 16 tokens s against this warp's 16; `odd`: on the diagonal, with values that are not finite.  (A form of its own: looked at
        // product by product it takes 13 % of the kernel.)
        auto weigh = [&](int ks, auto odd) {
            uint32_t pa[3][4];
            float pw[2][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = 2 * ks + half, s = t * 8 + q2;
                const float *lo = sD + (tw + g) * (C + 1) + s, *hi = lo + 8 * (C + 1);
                uint32_t w[3], x[3];
                // tokens after this one are left out, whatever their products are: zero times an infinity is none
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    pw[half][e] = s + (e & 1) <= tw + g + (e >> 1) * 8 ? qk[t][e] * (e < 2 ? lo : hi)[e & 1] : 0.f;
                ssd_split2(pw[half][0], pw[half][1], w);
                ssd_split2(pw[half][2], pw[half][3], x);
#pragma unroll
                for (int p = 0; p < 3; ++p) { pa[p][2 * half] = w[p]; pa[p][2 * half + 1] = x[p]; }
            }
#pragma unroll
            for (int pr = 0; pr < 4; ++pr) {
                uint32_t vb[4];
                ssd_ldm4t(vb, ssd_u32(sV) + ssd_at<8>(ks * 16 + (lm & 1) * 8 + lr, pr * 2 + (lm >> 1)));
                if constexpr (odd.value) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) vb[i] = ssd_finite(vb[i]);
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ssd_mma(o[2 * pr], pa[p], vb[0], vb[1]);
                    ssd_mma(o[2 * pr + 1], pa[p], vb[2], vb[3]);
                }
            }
            if constexpr (odd.value) {                       // the values left out, for their own and later tokens alone
#pragma unroll 1
                for (int s = 0; s < 16; ++s) {
                    const int from = (lane & 28) | ((s & 7) >> 1);
                    const float p0 = __shfl_sync(0xffffffffu, s & 8 ? (s & 1 ? pw[1][1] : pw[1][0]) : (s & 1 ? pw[0][1] : pw[0][0]), from);
                    const float p1 = __shfl_sync(0xffffffffu, s & 8 ? (s & 1 ? pw[1][3] : pw[1][2]) : (s & 1 ? pw[0][3] : pw[0][2]), from);
#pragma unroll
                    for (int x = 0; x < 8; ++x) {
                        const __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(sV + ssd_at<8>(ks * 16 + s, x) + q2 * 2);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float v = e ? __high2float(vv) : __low2float(vv);
                            if (isfinite(v)) continue;
                            if (s <= g) o[x][e] = fmaf(p0, v, o[x][e]);
                            if (s <= g + 8) o[x][2 + e] = fmaf(p1, v, o[x][2 + e]);
                        }
                    }
                }
            }
        };
        const bool odd = s_odd[warp];
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            if (ks > warp) continue;
            if (odd && ks == warp) weigh(ks, std::true_type{});
            else weigh(ks, std::false_type{});
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = tw + g + e * 8;
            if (t >= nt) continue;
            float* orow = a.out + (size_t)(r0 + t0 + t) * a.out_stride + (size_t)h * a.dv + j0;
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(sV + ssd_at<8>(t, x) + q2 * 2);
                *reinterpret_cast<float2*>(orow + x * 8 + q2) =
                    make_float2(fmaf(skip, __low2float(vv), o[x][2 * e] * a.q_scale), fmaf(skip, __high2float(vv), o[x][2 * e + 1] * a.q_scale));
            }
        }
        __syncthreads();                                     // q and the decays have been read
#pragma unroll 4
        for (int i = tid; i < C * P / 2; i += SSD_THREADS) { // the weighted values in three parts
            const int t = i / (P / 2), c = i % (P / 2);
            const uint32_t at = ssd_at<8>(t, c >> 2) + (c & 3) * 4;
            const __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(sV + at);
            uint32_t w[3];
            ssd_split2(__low2float(vv) * s_w[t], __high2float(vv) * s_w[t], w);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(sW + p * C * P * 2 + at) = w[p];
        }
        const float all = s_d0[C - 1];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < 8; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[m][t][e] *= all;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {                     // 16 tokens
            uint32_t ka[MT][4];
#pragma unroll
            for (int m = 0; m < MT; ++m)                     // K^T: stored by token, transposed on the way
                ssd_ldm4t(ka[m], ssd_u32(sK) + ssd_at<QR>(ks * 16 + (lm >> 1) * 8 + lr, (i0 + m * 16) / 8 + (lm & 1)));
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int pr = 0; pr < 4; ++pr) {
                    uint32_t wb[4];
                    ssd_ldm4t(wb, ssd_u32(sW) + p * C * P * 2 + ssd_at<8>(ks * 16 + (lm & 1) * 8 + lr, pr * 2 + (lm >> 1)));
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        ssd_mma(S[m][2 * pr], ka[m], wb[0], wb[1]);
                        ssd_mma(S[m][2 * pr + 1], ka[m], wb[2], wb[3]);
                    }
                }
        }
        __syncthreads();                                     // k, v and the weighted values have been read
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                *reinterpret_cast<float2*>(S_area + (size_t)(i0 + m * 16 + g + e * 8) * a.dv + t * 8 + q2) = make_float2(S[m][t][2 * e], S[m][t][2 * e + 1]);
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
                              float q_scale, void* stream) {
    if (n_seqs <= 0) return BRAID_OK;
    if (heads <= 0 || groups <= 0 || heads % groups) BRAID_REFUSE("ssd_scan: %d heads do not divide into %d groups", heads, groups);
    if ((dk != 64 && dk != 128) || dv <= 0 || dv % SSD_P) BRAID_REFUSE("ssd_scan: built for keys of 64 or 128 and values in multiples of 64, not %d x %d", dk, dv);
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) || q_stride % 8 || k_stride % 8 || v_stride % 8) BRAID_REFUSE("ssd_scan: rows must start on 16 bytes");
    if (((uintptr_t)out & 7) || out_stride % 2 || !state || (((uintptr_t)state | (uintptr_t)state_offset | (uintptr_t)state_stride) & 7)) BRAID_REFUSE("ssd_scan: results and state must start on 8 bytes");
    if (!gate_bias || !a_log || n_seqs > 65535 || dv / SSD_P > 65535) BRAID_REFUSE("ssd_scan: a bias and A_log are required, and the step must fit a launch");
    using B = const __nv_bfloat16*;
    SsdArgs a{(B)q, (B)k, (B)v, (B)gate, (B)gate_bias, (B)a_log, (B)skip, q_stride, k_stride, v_stride, gate_stride, out, out_stride,
              (uint8_t*)state, state_stride, state_offset, q_start, q_len, slot_ids, heads, groups, dv, q_scale};
    return dk == 64 ? launch_ssd<64>(a, n_seqs, (cudaStream_t)stream) : launch_ssd<128>(a, n_seqs, (cudaStream_t)stream);
}
