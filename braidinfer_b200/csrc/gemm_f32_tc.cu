// The 32-bit matrix product out[n, m] = sum_k x[n, k] * w[m, k] of prompts on the 5th-generation tensor cores: float32 operands as sums of
// three bfloat16 numbers (24 bits), of the nine products of their parts the six largest, float32 accumulation.  What is left out is below
// 2^-25 of |x w|, less than float32's rounding of one product.
//
// The tensor cores cut off where float32 rounds, so an accumulator in tensor memory holds 64 numbers of k at a time (the five small
// products first, then the first parts', four additions at the sum's own size) and is then added to the thread's float32 sums: measured
// beside float64 (k 1024 / 2816 / 4096) it is 1.1e-7 / 1.5e-7 / 1.7e-7 of the result's size off where gemm_tile_kernel is 2.9e-7 to 5.7e-7 /
// 4.8e-7 to 9.5e-7 / 5.7e-7 to 1.2e-6.  Below 2^-110 an operand's parts would fall under bfloat16's smallest exponent and lose its low bits
// (at 1e-37 all but 11), so operands are multiplied by 2^24 on their way: every float32 number is three parts then, and the results are 2^48
// too large until the end.  A result that is not finite (there: from 2^80 on) is worked out again by float32 multiply-adds, so that infinities and
// numbers whose parts or sums overflow do what they do there.
//
// A CTA of sixteen warps owns 128 weight rows x N tokens and walks k 64 at a time through two stages: while the tensor cores work on one, the
// warps fetch the next block's float32 numbers, read the accumulator of the block before, and split the numbers into the swizzled
// operand tiles of the other stage.  Bound by the splits and the barrier between two blocks (2.0 us a block of 64 with N = 128, of which the
// tensor cores work 12 N cycles, 0.8 us).  Measured beside gemm_tile_kernel (FFMA at 0.4 of its rate), L2 flushed, us: 480 tokens 1536 x 1024
// 33 / 75, 1024 x 1024 32 / 45, 5632 x 1024 79 / 175, 1024 x 2816 69 / 108; 2,048 tokens 5632 x 1024 183 / 633, 4096 x 4096 512 / 1,836; 17 tokens
// 1536 x 1024 30 / 43, 32768 x 1024 59 / 133, 200 x 516 21 / 27.  With 8 warps instead of 16 a CTA 2,048 tokens of 5632 x 1024 took 254 us where
// 16 took 187.
#include "tcgen05.cuh"

#define F3_BK 64
#define F3_BM 128
#define F3_THREADS 512
#define F3_UP 16777216.f                     // 2^24
#define F3_ROWS (F3_THREADS / 16)            // rows of 16 float4 that the CTA takes at once

struct GemmF32TcArgs {
    const float *x, *w, *res;
    float* out;
    int n_rows, m_out, k_in;
    long long ldx, ldw, ldo;
    int* error_flag;
};

template <int N> constexpr int f3_stage() { return 3 * (F3_BM + N) * F3_BK * 2; }
template <int N> constexpr int f3_smem() { return 2 * f3_stage<N>() + 1024; }
template <int N> constexpr uint32_t f3_cols() { return N <= 32 ? 64 : N <= 64 ? 128 : 256; }      // two accumulators, a power of two

// F3_UP times two numbers
__device__ __forceinline__ uint64_t f3_scaled(float a, float b) {
    uint64_t v;
    asm("{\n\t.reg .b64 x, up;\n\tmov.b64 x, {%1, %2};\n\tmov.b64 up, {%3, %3};\n\tmul.rn.f32x2 %0, x, up;\n\t}" : "=l"(v) : "f"(a), "f"(b), "f"(F3_UP));
    return v;
}
// four numbers to their places in three operand tiles of `part` bytes: 128-byte rows, 16-byte runs swapped by the row's low bits
__device__ __forceinline__ void f3_split(uint32_t tile, uint32_t part, int r, int c, float4 x) {
    const uint32_t at = tile + r * 128 + (((c >> 1) ^ (r & 7)) << 4) + (c & 1) * 8;
    uint64_t v[2] = {f3_scaled(x.x, x.y), f3_scaled(x.z, x.w)};      // two numbers a register pair and instruction
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint32_t w[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float a, b;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v[e]));
            // (the first two saturate: a number past the largest bfloat16 one is still a sum of finite parts)
            if (p < 2) {
                asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w[e]) : "f"(b), "f"(a));
                uint64_t part;
                asm("mov.b64 %0, {%1, %2};" : "=l"(part) : "r"(w[e] << 16), "r"(w[e] & 0xffff0000u));
                asm("sub.rn.f32x2 %0, %0, %1;" : "+l"(v[e]) : "l"(part));
            } else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[e]) : "f"(b), "f"(a));
        }
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + p * part), "r"(w[0]), "r"(w[1]) : "memory");
    }
}

template <int N>
__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ GemmF32TcArgs a) {
    constexpr int NA = F3_BM / F3_ROWS, NB = N / F3_ROWS;                            // float4 a thread and block of A, of B
    constexpr int DW = N % 64 ? 8 : 16, COLS = N / (DW / 4);                         // warps that read accumulators, columns each
    static_assert(COLS % 16 == 0 && N % F3_ROWS == 0, "whole loads");
    constexpr uint32_t PA = F3_BM * F3_BK * 2, PB = N * F3_BK * 2;
    extern __shared__ uint8_t f3_raw[];
    __shared__ uint64_t done[2];
    __shared__ uint32_t slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const uint32_t base = (smem_u32(f3_raw) + 1023u) & ~1023u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * F3_BM, n0 = blockIdx.y * N;
    pdl_trigger();
    if (tid == 0) {
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&slot, f3_cols<N>());
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = slot;
    const int r0 = tid >> 4, c = tid & 15;
    float4 av[2][NA], bv[2][NB];                             // two blocks on their way
    auto fetch_w = [&](float4* av, int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int m = m0 + r0 + i * F3_ROWS, k = k0 + c * 4;
            av[i] = m < a.m_out && k < a.k_in ? *reinterpret_cast<const float4*>(a.w + (size_t)m * a.ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto fetch_x = [&](float4* bv, int k0) {
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int n = n0 + r0 + i * F3_ROWS, k = k0 + c * 4;
            bv[i] = n < a.n_rows && k < a.k_in ? *reinterpret_cast<const float4*>(a.x + (size_t)n * a.ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    float acc[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
    const uint32_t mine = tmem + ((uint32_t)(warp & 3) * 32 << 16) + (warp >> 2) * COLS;
    auto drain = [&](int kb) {
        mbar_wait(&done[kb & 1], (kb >> 1) & 1, abort_flag);         // (every warp: the stage's next numbers are written after it)
        if (warp >= DW) return;
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < COLS; j += 16) {
            float v[16];
            tmem_ld16(mine + (kb & 1) * N + j, v);
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[j + e] += v[e];
        }
        tc_fence_before();
    };
    const int blocks = (a.k_in + F3_BK - 1) / F3_BK;
    fetch_w(av[0], 0);
    fetch_w(av[1], F3_BK);
    pdl_wait();
    fetch_x(bv[0], 0);
    fetch_x(bv[1], F3_BK);
#pragma unroll 1
    for (int k2 = 0; k2 < blocks; k2 += 2)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int kb = k2 + b;
            if (kb >= blocks) break;
            const uint32_t sa = base + b * f3_stage<N>(), sb = sa + 3 * PA;      // read by the block two before, which has been drained
#pragma unroll
            for (int i = 0; i < NA; ++i) f3_split(sa, PA, r0 + i * F3_ROWS, c, av[b][i]);
#pragma unroll
            for (int i = 0; i < NB; ++i) f3_split(sb, PB, r0 + i * F3_ROWS, c, bv[b][i]);
            if (kb + 2 < blocks) {
                fetch_w(av[b], (kb + 2) * F3_BK);
                fetch_x(bv[b], (kb + 2) * F3_BK);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                const uint32_t idesc = umma_idesc_bf16(F3_BM, N), d = tmem + b * N;
                const uint64_t da = umma_desc_sw128(sa), db = umma_desc_sw128(sb);         // (addresses in units of 16 bytes in the low bits)
                constexpr int pa[6] = {1, 0, 2, 0, 1, 0}, pb[6] = {1, 2, 0, 1, 0, 0};      // the small products first
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < F3_BK / 16; ++k)
                        umma_bf16(d, da + (pa[p] * PA + k * 32) / 16, db + (pb[p] * PB + k * 32) / 16, idesc, p + k > 0);
                umma_commit(&done[b]);
            }
            if (kb > 0) drain(kb - 1);
        }
    drain(blocks - 1);
    const int m = m0 + (warp & 3) * 32 + lane;
    if (warp < DW && m < a.m_out && !*abort_flag)
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            const int n = n0 + (warp >> 2) * COLS + j;
            if (n >= a.n_rows) break;
            float v = acc[j] * (1.f / F3_UP / F3_UP);
            if (!(fabsf(v) <= 3.402823466e38f)) {
                v = 0.f;
                for (int k = 0; k < a.k_in; ++k) v = fmaf(a.x[(size_t)n * a.ldx + k], a.w[(size_t)m * a.ldw + k], v);
            }
            const size_t at = (size_t)n * a.ldo + m;
            a.out[at] = a.res ? a.res[at] + v : v;
        }
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(a.error_flag, 1);
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, f3_cols<N>());
    }
}

template <int N>
static int launch_f3(const GemmF32TcArgs& a, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, f3_smem<N>());
        if (e != cudaSuccess) { braid_set_error("gemm_f32_tc: cannot reserve %d bytes of shared memory: %s", f3_smem<N>(), cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    braid_launch(gemm_f32_tc_kernel<N>, dim3((a.m_out + F3_BM - 1) / F3_BM, (a.n_rows + N - 1) / N), dim3(F3_THREADS), (size_t)f3_smem<N>(), s, a);
    BRAID_LAUNCH_CHECK();
}

// float32 operands whose rows start on 16 bytes, k a multiple of 4.  res (may be out): out = res + product.
extern "C" int braid_gemm_f32_tc(const float* x, const float* w, float* out, const float* res, int n_rows, int m_out, int k_in, long long ldx,
                                 long long ldw, long long ldo, int* error_flag, void* stream) {
    if (n_rows <= 0 || m_out <= 0) return BRAID_OK;
    if (k_in <= 0 || k_in % 4 || ldx % 4 || ldw % 4 || (((uintptr_t)x | (uintptr_t)w) & 15)) BRAID_REFUSE("gemm_f32_tc: rows must start on 16 bytes, k=%d must be a multiple of 4", k_in);
    if (!error_flag) BRAID_REFUSE("gemm_f32_tc: error_flag is required");
    if (n_rows > 65535 * 32) BRAID_REFUSE("gemm_f32_tc: %d rows exceed the grid limit", n_rows);
    const GemmF32TcArgs a{x, w, res, out, n_rows, m_out, k_in, ldx, ldw, ldo, error_flag};
    // the token tile with the fewest numbers to split on the busiest SM (each tile costs its 128 weight rows again, and some 64 rows' worth
    // of barriers)
    int best = 0;
    long long least = 0;
    for (int n = 32; n <= 128; n += 32) {
        const long long tiles = (long long)((m_out + F3_BM - 1) / F3_BM) * ((n_rows + n - 1) / n), cost = (tiles + 147) / 148 * (F3_BM + 64 + n);
        if (!best || cost < least) { best = n; least = cost; }
    }
    cudaStream_t s = (cudaStream_t)stream;
    return best == 32 ? launch_f3<32>(a, s) : best == 64 ? launch_f3<64>(a, s) : best == 96 ? launch_f3<96>(a, s) : launch_f3<128>(a, s);
}
