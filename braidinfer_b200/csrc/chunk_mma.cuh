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
// Inside a sub-chunk of 16 the decay from s to t is (start to t) (s to end) / (start to end).  The factors stay normal numbers, and what
// is lost of the smallest is far below a sum's rounding, while a channel's decays over the sub-chunk multiply to 2^-100 or more; the
// channels beyond are steep and multiplied up pair by pair.
#define CHK_SPREAD 7.8886091e-31f          // 2^-100
// Queries and keys that are decayed that far stay normal numbers, and hold three parts of bfloat16 (which ends at 2^-133), down to 2^-60 in
// size because both are stored times CHK_UP; the scores' products lie between 2^-50 and 2^50 of their queries and keys, and fit up to CHK_LARGE.
// Decays above one are taken as others while they multiply to CHK_GROWTH or less.  (Elsewhere an operand that has decayed below 2^-110 stands in
// a sum beside ones that have not; what it loses is 2^-134 of the other factor.)
#define CHK_UP 1.125899906842624e15f       // 2^50
#define CHK_LARGE 274877906944.f           // 2^38
#define CHK_GROWTH 1048576.f               // 2^20
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

// Four neighbouring numbers as float32, one by one where they do not start on 16 (8) bytes.
__device__ __forceinline__ float4 chk_load4(const float* p, bool wide) {
    return wide ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
// Eight neighbouring bfloat16 numbers as they lie.
__device__ __forceinline__ uint4 chk_load8(const __nv_bfloat16* p, bool wide) {
    if (wide) return *reinterpret_cast<const uint4*>(p);
    const uint16_t* s = reinterpret_cast<const uint16_t*>(p);
    return make_uint4(s[0] | (uint32_t)s[1] << 16, s[2] | (uint32_t)s[3] << 16, s[4] | (uint32_t)s[5] << 16, s[6] | (uint32_t)s[7] << 16);
}

// A channel's decays over a sub-chunk, by the thread that owns the two: `d` [16 rows of LD] holds the decays and gets the products from the
// sub-chunk's start on; `k` is decayed to its end and, where asked for, `f` is k decayed from its start, both times CHK_UP.  True: a steep
// channel.
template <int LD, bool FORWARD>
__device__ __forceinline__ bool chk_decays(float* d, float* k, float* f, float* total, float* inv) {
    float dec[CHK_SUB], prod = 1.f, after = CHK_UP;
#pragma unroll
    for (int r = 0; r < CHK_SUB; ++r) dec[r] = d[r * LD];
#pragma unroll
    for (int r = 0; r < CHK_SUB; ++r) {
        prod *= dec[r];
        d[r * LD] = prod;
        if (FORWARD) f[r * LD] = k[r * LD] * (prod * CHK_UP);
    }
#pragma unroll
    for (int r = CHK_SUB - 1; r >= 0; --r) {
        k[r * LD] *= after;
        after *= dec[r];
    }
    const bool steep = !(prod >= CHK_SPREAD && prod <= CHK_GROWTH);
    *total = prod;
    *inv = steep ? 0.f : (1.f / CHK_UP / CHK_UP) / prod;
    return steep;
}

// Products of a block of 16 rows (decayed from their sub-chunk's start) with the keys (decayed to their sub-chunk's end) of the same
// sub-chunk J and the ones before it: acc[d] for sub-chunk J - d, TILES tiles of 8 keys from tile0 on, in mma.sync's layout; the products of
// the first parts, and the small ones.  Between two sub-chunks lie the decays of those between; inside one, 1 / all of its decays.
// Rows and keys are CHK_UP times theirs, the results are not.
template <int DK, int LD, int TILES>
__device__ __forceinline__ void chk_scores(const float* rows, const float* keys, const float* total, const float* inv, int J, int tile0,
                                           float (*acc)[TILES][2][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q2 = (lane & 3) * 2;
#pragma unroll
    for (int d = 0; d < 4; ++d)
#pragma unroll
        for (int x = 0; x < TILES; ++x)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[d][x][e >> 2][e & 3] = 0.f;
#pragma unroll 1
    for (int c = q2; c < DK; c += 16) {                      // channels c, c + 1, c + 8, c + 9
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 v = *reinterpret_cast<const float2*>(rows + (g + (e & 1) * 8) * LD + c + (e >> 1) * 8);
            chk_split2(v.x, v.y, a[0][e], a[1][e], a[2][e]);
        }
        float2 f[2] = {make_float2(1.f / CHK_UP, 1.f / CHK_UP), make_float2(1.f / CHK_UP, 1.f / CHK_UP)};
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            if (d > J) continue;
            const int I = J - d;
            if (d > 1) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const float2 t = *reinterpret_cast<const float2*>(total + (I + 1) * DK + c + w * 8);
                    f[w].x *= t.x;
                    f[w].y *= t.y;
                }
            }
            uint32_t b[TILES][3][2];
#pragma unroll
            for (int x = 0; x < TILES; ++x)
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    float2 v = *reinterpret_cast<const float2*>(keys + (I * CHK_SUB + (tile0 + x) * 8 + g) * LD + c + w * 8);
                    const float2 m = d == 0 ? *reinterpret_cast<const float2*>(inv + J * DK + c + w * 8) : f[w];
                    chk_split2(v.x * m.x, v.y * m.y, b[x][0][w], b[x][1][w], b[x][2][w]);
                }
            CHK_PAIRS(3, 3, pa, pb) {
#pragma unroll
                for (int x = 0; x < TILES; ++x)
                    if (pa + pb == 0) chk_mma_sum<true>(acc[d][x], a[pa], b[x][pb][0], b[x][pb][1]);
                    else chk_mma_sum<false>(acc[d][x], a[pa], b[x][pb][0], b[x][pb][1]);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 4; ++d)
#pragma unroll
        for (int x = 0; x < TILES; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[d][x][0][e] = (acc[d][x][0][e] + acc[d][x][1][e]) * (d == 0 ? 1.f : 1.f / CHK_UP);
}

// The steep channels' share of the blocks on the diagonal, pair by pair: for every sub-chunk J, `take(J, p, a)` after the sums of q_t k_s and
// (BOTH) k_t k_s lie in p and a [16][17].  `inv` [4][DK] is 0 for a steep channel of a sub-chunk; `stage`: CHK_STEEP_FLOATS(DK) floats
// that nobody else needs between the barriers around the call; q, k and decay of (token, channel) come from the caller.
#define CHK_STEEP_FLOATS(DK) (3 * CHK_SUB * (DK) + 2 * CHK_SUB * 17)
template <int DK, bool BOTH, typename Q, typename K, typename D, typename Take>
__device__ __forceinline__ void chk_steep(float* stage, const float* inv, int n, Q q, K k, D decay, Take take) {
    constexpr int SUB = CHK_SUB;
    __shared__ uint32_t mask[DK / 32];
    float *sG = stage, *sK = sG + SUB * DK, *sQ = sK + SUB * DK, *sP = sQ + SUB * DK, *sA = sP + SUB * 17;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
#pragma unroll 1
    for (int J = 0; J < 4; ++J) {
        if (tid < DK) {
            const uint32_t m = __ballot_sync(0xffffffffu, inv[J * DK + tid] == 0.f);
            if ((tid & 31) == 0) mask[tid >> 5] = m;
        }
#pragma unroll 1
        for (int idx = tid; idx < SUB * DK; idx += CHK_THREADS) {
            const int r = idx / DK, i = idx % DK, t = J * SUB + r;
            const bool in = t < n && inv[J * DK + i] == 0.f;
            sG[idx] = in ? decay(t, i) : 1.f;
            sK[idx] = in ? k(t, i) : 0.f;
            sQ[idx] = in ? q(t, i) : 0.f;
        }
        __syncthreads();
        float p = 0.f, a = 0.f;
        if (tx <= ty)
            for (int w = 0; w < DK / 32; ++w)
                for (uint32_t m = mask[w]; m; m &= m - 1) {
                    const int i = w * 32 + __ffs(m) - 1;
                    float x = sK[tx * DK + i];
                    for (int r = tx + 1; r <= ty; ++r) x *= sG[r * DK + i];
                    p = fmaf(sQ[ty * DK + i], x, p);
                    if (BOTH) a = fmaf(sK[ty * DK + i], x, a);
                }
        sP[ty * 17 + tx] = p;
        if (BOTH) sA[ty * 17 + tx] = a;
        __syncthreads();
        take(J, sP, sA);
    }
    __syncthreads();
}

// The outputs of 64 tokens x NB value columns by 256 threads: MW warps along the tokens, the others along the columns, 16 columns a warp.
// The state's numbers go from memory straight into operand registers, each read by MW warps: `fetch(x, ks)` brings, for keys
// ks * 16 + lq, + 1, + 8, + 9, those of the warp's columns lg (x[0 ..]) and lg + 8 (x[4 ..]), lane = lg * 4 + lq / 2.  `stage(place)` brings
// what the values need to shared memory, `values(b, ks, place)` their operands of 16 tokens in PV parts.  `store(token, column of the CTA, x, y)`
// takes two neighbouring results.  With WALK, true for the whole CTA: a number of the state is not finite, or `odd`; nothing was stored.
template <int DK, int STAGE> constexpr int chk_out_smem() { return (3 * CHK_C * (DK + 8) + 3 * CHK_C * CHK_PPITCH) * 2 + STAGE; }
template <int NB> __device__ __forceinline__ int chk_out_col() { return (threadIdx.x >> 5) % (NB / 16) * 16; }      // the warp's first column
template <int DK, int PV, int NB, bool WALK, typename Fetch, typename Stage, typename Values, typename Store>
__device__ __forceinline__ bool chk_outputs(void* smem, const float* __restrict__ gq, const float* __restrict__ gp, bool odd, Fetch fetch, Stage stage,
                                            Values values, Store store) {
    constexpr int C = CHK_C, NT = CHK_THREADS, QP = DK + 8;
    constexpr int CW = NB / 16, MW = 8 / CW, MT = 4 / MW;    // warps along the columns, along the tokens; tiles of 16 tokens a warp
    __nv_bfloat16* sQ = (__nv_bfloat16*)smem;                // 3 x [C][QP]
    __nv_bfloat16* sP = sQ + 3 * C * QP;                     // 3 x [C][CHK_PPITCH]
    __nv_bfloat16* place = sP + 3 * C * CHK_PPITCH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lq = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    const int cw = warp % CW * 16, mw = warp / CW * MT;
    constexpr int AHEAD = 2;
    float sv[AHEAD][8];
#pragma unroll
    for (int ks = 0; ks < AHEAD; ++ks) fetch(sv[ks], ks);
    stage(place);
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
        values(vb, ks, place);
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
                store((mw + m) * 16 + lg + e * 8, cw + lq + x * 8, o[m][x][0][2 * e] + o[m][x][1][2 * e],
                      o[m][x][0][2 * e + 1] + o[m][x][1][2 * e + 1]);
    return false;
}
