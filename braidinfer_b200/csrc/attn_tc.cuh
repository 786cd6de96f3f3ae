// Inline-PTX wrappers shared by the prompt-attention kernels on tcgen05: tensor-memory loads and stores of 64 columns,
// tcgen05.mma with operand descriptors in two words and with the A operand in tensor memory.
#pragma once
#include "tcgen05.cuh"

#define FA_RAISE 8.f                             // how far a tile's maximum may exceed m before m is raised

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));       // exp2(-inf) = 0, exp2(0) = 1 exactly
    return y;
}
// 64 consecutive columns of this thread's lane: two loads in flight, one wait.
__device__ __forceinline__ void tmem_ld32x2(uint32_t taddr, float* v) {
    uint32_t r[64];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[h * 32 + 0]), "=r"(r[h * 32 + 1]), "=r"(r[h * 32 + 2]), "=r"(r[h * 32 + 3]), "=r"(r[h * 32 + 4]),
              "=r"(r[h * 32 + 5]), "=r"(r[h * 32 + 6]), "=r"(r[h * 32 + 7]), "=r"(r[h * 32 + 8]), "=r"(r[h * 32 + 9]),
              "=r"(r[h * 32 + 10]), "=r"(r[h * 32 + 11]), "=r"(r[h * 32 + 12]), "=r"(r[h * 32 + 13]), "=r"(r[h * 32 + 14]),
              "=r"(r[h * 32 + 15]), "=r"(r[h * 32 + 16]), "=r"(r[h * 32 + 17]), "=r"(r[h * 32 + 18]), "=r"(r[h * 32 + 19]),
              "=r"(r[h * 32 + 20]), "=r"(r[h * 32 + 21]), "=r"(r[h * 32 + 22]), "=r"(r[h * 32 + 23]), "=r"(r[h * 32 + 24]),
              "=r"(r[h * 32 + 25]), "=r"(r[h * 32 + 26]), "=r"(r[h * 32 + 27]), "=r"(r[h * 32 + 28]), "=r"(r[h * 32 + 29]),
              "=r"(r[h * 32 + 30]), "=r"(r[h * 32 + 31])
            : "r"(taddr + h * 32) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}
// tcgen05.mma with both operands in shared memory, and with the A operand in tensor memory (rows in
// lanes, K packed two bfloat16 a column).  Descriptors are given as (low word, high word): a
// descriptor's start address lives in its low word, the high word is the same for all tiles of a kind.
__device__ __forceinline__ void umma_ss_lohi(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_ts_lohi(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_addr(uint32_t bar_addr) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_addr) : "memory");
}
// 32 consecutive columns of this thread's lane written (no wait).
__device__ __forceinline__ void tmem_st32_nowait(uint32_t taddr, const uint32_t* w) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        :: "r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]),
           "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]),
           "r"(w[18]), "r"(w[19]), "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(w[24]), "r"(w[25]), "r"(w[26]),
           "r"(w[27]), "r"(w[28]), "r"(w[29]), "r"(w[30]), "r"(w[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The reverse: 64 consecutive columns of this thread's lane written back.
__device__ __forceinline__ void tmem_st32x2(uint32_t taddr, const float* v) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
            "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
            :: "r"(taddr + h * 32),
               "r"(__float_as_uint(v[h * 32 + 0])), "r"(__float_as_uint(v[h * 32 + 1])), "r"(__float_as_uint(v[h * 32 + 2])),
               "r"(__float_as_uint(v[h * 32 + 3])), "r"(__float_as_uint(v[h * 32 + 4])), "r"(__float_as_uint(v[h * 32 + 5])),
               "r"(__float_as_uint(v[h * 32 + 6])), "r"(__float_as_uint(v[h * 32 + 7])), "r"(__float_as_uint(v[h * 32 + 8])),
               "r"(__float_as_uint(v[h * 32 + 9])), "r"(__float_as_uint(v[h * 32 + 10])), "r"(__float_as_uint(v[h * 32 + 11])),
               "r"(__float_as_uint(v[h * 32 + 12])), "r"(__float_as_uint(v[h * 32 + 13])), "r"(__float_as_uint(v[h * 32 + 14])),
               "r"(__float_as_uint(v[h * 32 + 15])), "r"(__float_as_uint(v[h * 32 + 16])), "r"(__float_as_uint(v[h * 32 + 17])),
               "r"(__float_as_uint(v[h * 32 + 18])), "r"(__float_as_uint(v[h * 32 + 19])), "r"(__float_as_uint(v[h * 32 + 20])),
               "r"(__float_as_uint(v[h * 32 + 21])), "r"(__float_as_uint(v[h * 32 + 22])), "r"(__float_as_uint(v[h * 32 + 23])),
               "r"(__float_as_uint(v[h * 32 + 24])), "r"(__float_as_uint(v[h * 32 + 25])), "r"(__float_as_uint(v[h * 32 + 26])),
               "r"(__float_as_uint(v[h * 32 + 27])), "r"(__float_as_uint(v[h * 32 + 28])), "r"(__float_as_uint(v[h * 32 + 29])),
               "r"(__float_as_uint(v[h * 32 + 30])), "r"(__float_as_uint(v[h * 32 + 31]))
            : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
