// What the recurrences over chunks of 64 tokens share (scan_chunk.cu, delta_chunk.cu): float32 operands of mma.sync as sums of three
// bfloat16 numbers, and the outputs of a chunk,
//   O = Q S_0 + P V,
// Q [64][dk] (queries decayed from the chunk's start), P [64][64] (lower triangular), S_0 [dk][dv], all float32.
//
// x = x0 + x1 + x2 holds float32's 24 bits; of the products of two such sums the six largest are taken, what is left out is of the size of
// float32's own rounding.  The tensor cores cut off where float32 rounds, so the products of the first parts, which carry the size of the
// sum, are added up by float32 additions, 16 of k at a time, and only the small ones in the tensor cores' accumulators (all there: four
// times the error of the walk token by token; the first parts in accumulators of their own: twice).
#pragma once
#include "common.cuh"

#define CHK_C 64
#define CHK_SUB 16
#define CHK_THREADS 256
#define CHK_SPREAD 8.6736174e-19f          // 2^-60
#define CHK_PPITCH (CHK_C + 8)

__device__ __forceinline__ bool chk_not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }
__device__ __forceinline__ uint32_t chk_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void chk_ldm4(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void chk_ldm4t(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void chk_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += a b with float32's rounding of the sum; or in the tensor cores' accumulator
template <bool FIRST>
__device__ __forceinline__ void chk_mma_sum(float (*c)[4], const uint32_t* a, uint32_t b0, uint32_t b1) {
    if (!FIRST) return chk_mma(c[1], a, b0, b1);
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    chk_mma(t, a, b0, b1);
#pragma unroll
    for (int e = 0; e < 4; ++e) c[0][e] += t[e];
}
// The three parts of x0 and x1, packed (x0 in the low half).  The first two saturate, so that a number past the largest bfloat16 one is
// still a sum of finite parts.
__device__ __forceinline__ void chk_split2(float x0, float x1, uint32_t& w0, uint32_t& w1, uint32_t& w2) {
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w0) : "f"(x1), "f"(x0));
    x0 -= __uint_as_float(w0 << 16);
    x1 -= __uint_as_float(w0 & 0xffff0000u);
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w1) : "f"(x1), "f"(x0));
    x0 -= __uint_as_float(w1 << 16);
    x1 -= __uint_as_float(w1 & 0xffff0000u);
    const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
    w2 = *reinterpret_cast<const uint32_t*>(&h);
}
// Four numbers to three places, `part` elements apart.
__device__ __forceinline__ void chk_store_split4(__nv_bfloat16* at, int part, float4 x) {
    uint32_t w[2][3];
    chk_split2(x.x, x.y, w[0][0], w[0][1], w[0][2]);
    chk_split2(x.z, x.w, w[1][0], w[1][1], w[1][2]);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * part) = make_uint2(w[0][p], w[1][p]);
}
// Operands of PA and PB parts: the pairs whose product is not below 2^-16 of the first parts'.
#define CHK_PAIRS(PA, PB, pa, pb) _Pragma("unroll") for (int pa = 0; pa < PA; ++pa) _Pragma("unroll") for (int pb = 0; pb < PB; ++pb) if (pa + pb <= 2)

// The outputs of 64 tokens x NB value columns by 256 threads: MW warps along the tokens, the others along the columns, 16 columns a warp.
// The state's numbers go from memory straight into operand registers, each read by MW warps.  V has PV parts (1: bfloat16 numbers as they
// are); `stage_v(dst, pitch, part)` brings its 64 rows to shared memory.  `store(token, column, x, y)` takes two neighbouring results.
// With WALK, true for the whole CTA: a number of the state is not finite, or `odd`; nothing was stored.
template <int DK, int PV, int NB> constexpr int chk_out_smem() {
    return (3 * CHK_C * (DK + 8) + 3 * CHK_C * CHK_PPITCH + PV * CHK_C * (NB + 8)) * 2;
}
template <int DK, int PV, int NB, bool WALK, typename StageV, typename Store>
__device__ __forceinline__ bool chk_outputs(void* smem, const float* __restrict__ gq, const float* __restrict__ gp, const float* __restrict__ S,
                                            int dv, int col0, bool odd, StageV stage_v, Store store) {
    constexpr int C = CHK_C, NT = CHK_THREADS, QP = DK + 8, VP = NB + 8;
    constexpr int CW = NB / 16, MW = 8 / CW, MT = 4 / MW;    // warps along the columns, along the tokens; tiles of 16 tokens a warp
    __nv_bfloat16* sQ = (__nv_bfloat16*)smem;                // 3 x [C][QP]
    __nv_bfloat16* sP = sQ + 3 * C * QP;                     // 3 x [C][CHK_PPITCH]
    __nv_bfloat16* sV = sP + 3 * C * CHK_PPITCH;             // PV x [C][VP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lq = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    const int cw = warp % CW * 16, mw = warp / CW * MT;
    const float* sp = S + (size_t)lq * dv + col0 + cw + lg;
    constexpr int AHEAD = 2;
    float sv[AHEAD][8];
    auto fetch = [&](float* x, int ks) {                     // keys ks * 16 + lq, + 1, + 8, + 9; columns lg and lg + 8
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float* at = sp + (size_t)(ks * 16 + (e & 1) + (e >> 1) * 8) * dv;
            x[e] = at[0];
            x[4 + e] = at[8];
        }
    };
#pragma unroll
    for (int ks = 0; ks < AHEAD; ++ks) fetch(sv[ks], ks);
    stage_v(sV, VP, C * VP);
#pragma unroll 4
    for (int idx = tid * 4; idx < C * DK; idx += NT * 4)
        chk_store_split4(sQ + idx / DK * QP + idx % DK, C * QP, *reinterpret_cast<const float4*>(gq + idx));
#pragma unroll
    for (int u = 0; u < C * C / 4 / NT; ++u) {
        const int idx = (tid + u * NT) * 4, t = idx / C, s = idx % C;
        const bool in = s / CHK_SUB <= t / CHK_SUB;          // the blocks beyond were not written
        chk_store_split4(sP + t * CHK_PPITCH + s, C * CHK_PPITCH, in ? *reinterpret_cast<const float4*>(gp + idx) : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    __syncthreads();
    float o[MT][2][2][4];                                    // the products of the first parts, and the small ones
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 8; ++e) o[m][x][e >> 2][e & 3] = 0.f;
    bool bad = odd;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
        uint32_t sb[2][3][2];
        float* x = sv[ks % AHEAD];
#pragma unroll
        for (int e = 0; e < 8; ++e) bad |= WALK && chk_not_finite(x[e]);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) chk_split2(x[t * 4 + e * 2], x[t * 4 + e * 2 + 1], sb[t][0][e], sb[t][1][e], sb[t][2][e]);
        if (ks + AHEAD < DK / 16) fetch(x, ks + AHEAD);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            uint32_t qa[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p)
                chk_ldm4(qa[p], chk_u32(sQ + p * C * QP + ((mw + m) * 16 + (lm & 1) * 8 + lr) * QP + ks * 16 + (lm >> 1) * 8));
            CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (pa + pb == 0) chk_mma_sum<true>(o[m][t], qa[pa], sb[t][pb][0], sb[t][pb][1]);
                    else chk_mma_sum<false>(o[m][t], qa[pa], sb[t][pb][0], sb[t][pb][1]);
            }
        }
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        uint32_t vb[PV][4];
#pragma unroll
        for (int p = 0; p < PV; ++p) chk_ldm4t(vb[p], chk_u32(sV + p * C * VP + (ks * 16 + (lm & 1) * 8 + lr) * VP + cw + (lm >> 1) * 8));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (ks > mw + m) continue;
            uint32_t pw[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p)
                chk_ldm4(pw[p], chk_u32(sP + p * C * CHK_PPITCH + ((mw + m) * 16 + (lm & 1) * 8 + lr) * CHK_PPITCH + ks * 16 + (lm >> 1) * 8));
            CHK_PAIRS(3, PV, pa, pb) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (pa + pb == 0) chk_mma_sum<true>(o[m][t], pw[pa], vb[pb][2 * t], vb[pb][2 * t + 1]);
                    else chk_mma_sum<false>(o[m][t], pw[pa], vb[pb][2 * t], vb[pb][2 * t + 1]);
            }
        }
    }
    if (WALK && __syncthreads_or(bad)) return true;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int x = 0; x < 2; ++x)
                store((mw + m) * 16 + lg + e * 8, col0 + cw + lq + x * 8, o[m][x][0][2 * e] + o[m][x][1][2 * e],
                      o[m][x][0][2 * e + 1] + o[m][x][1][2 * e + 1]);
    return false;
}
