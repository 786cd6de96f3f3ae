// Plain matrix product on the CUDA cores: out[n, m] = sum_k x[n, k] * w[m, k].
//
// w is [out_features, in_features] row-major as model folders store it, so y = W x
// (kernels/megakernel_ops.hip:168-216 of the reference; oracle
// crates/braidinfer-runtime/tests/linear_proj_test.rs:13-23).  Products and sums are
// IEEE float32 FMA in a fixed order along k; no tensor cores and no reduced-precision
// mode, which makes this the matrix product of the true 32-bit path (of more than 16 tokens where
// gemm_f32_tc.cu does not pay).  With bfloat16
// inputs it is the reference that the tensor-core kernel is checked against.
//
// Epilogues: 0 stores the product in `out_dtype`; 1 stores res + product as float32
// (the residual sum; out may be res itself).
#include "common.cuh"

#define SG_BM 64   // output features per block
#define SG_BN 64   // tokens per block
#define SG_BK 16

template <typename T, typename TO, int MODE>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ x, const T* __restrict__ w, TO* __restrict__ out,
                 const float* __restrict__ res, int n_rows, int m_out, int k_in,
                 long long ldx, long long ldw, long long ldo) {
    pdl_trigger();
    pdl_wait();
    __shared__ float xs[SG_BK][SG_BN + 4];
    __shared__ float ws[SG_BK][SG_BM + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;     // tx: outputs, ty: tokens
    const int n0 = blockIdx.y * SG_BN, m0 = blockIdx.x * SG_BM;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < k_in; k0 += SG_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 256;        // 0..1023
            const int r = e >> 4, c = e & 15;           // r: row in tile, c: k offset
            const int k = k0 + c;
            const int n = n0 + r, m = m0 + r;
            xs[c][r] = (n < n_rows && k < k_in) ? to_f32(x[(size_t)n * ldx + k]) : 0.f;
            ws[c][r] = (m < m_out && k < k_in) ? to_f32(w[(size_t)m * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < SG_BK; ++kk) {
            float xv[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int n = n0 + ty * 4 + i;
        if (n >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + tx * 4 + j;
            if (m >= m_out) continue;
            const size_t o = (size_t)n * ldo + m;
            if (MODE == 1) out[o] = from_f32<TO>(res[o] + acc[i][j]);
            else out[o] = from_f32<TO>(acc[i][j]);
        }
    }
}

// ------------------------------------------------------------------ the 32-bit path's products
// float32 rows and weights that can be read 16 bytes at a time take one of two kernels; the one above keeps the rest (and the
// bfloat16 twin).  Both are IEEE float32 FMA: only the order of the sums along k differs between them, and it depends on
// the product's sizes alone.
//
// A few rows (SK_MAX_ROWS): bound by the weights' bytes.  A warp owns four weight rows and up to eight tokens, its lanes
// stride along k with 16-byte loads; KS warps of a CTA share four rows' k where the rows alone would leave SMs idle, and
// their sums meet in shared memory in the warps' order.  (The kernel above walks k in dependent steps of 16 with one CTA for 64
// weight rows.)  All products of a four-layer decoder of width 1024, a prompt of 480 rows and 8 steps of 3, took 23.8 ms
// with the kernel above and take 2.5 with these two: 0.12 ms a step, 1.5 the prompt.
#define SK_WARPS 8
#define SK_MR 4
#define SK_MAX_ROWS 16

// The sums over a warp's lanes of V numbers a lane (V a power of two up to 32): lane l returns that of number
// l >> (5 - log2 V).
template <int V>
__device__ __forceinline__ float warp_sums(float* v) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = V; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float r = v[0];
#pragma unroll
    for (; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}

template <int N>
__global__ void __launch_bounds__(SK_WARPS * 32)
gemm_few_kernel(const float* __restrict__ x, const float* __restrict__ w, float* out, const float* res, int n_rows, int m_out,
                int k4, int ks, long long ldx, long long ldw, long long ldo) {
    constexpr int V = SK_MR * N, U = 2;
    constexpr int SHIFT = V == 4 ? 3 : V == 8 ? 2 : V == 16 ? 1 : 0;
    __shared__ float part[SK_WARPS][V];
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = SK_WARPS / ks, group = warp / ks, slice = warp - group * ks;
    const int m0 = (blockIdx.x * groups + group) * SK_MR, n0 = blockIdx.y * N;
    const float4* wr[SK_MR];
#pragma unroll
    for (int r = 0; r < SK_MR; ++r) wr[r] = reinterpret_cast<const float4*>(w + (size_t)min(m0 + r, m_out - 1) * ldw);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int step = ks * 32;
    int i = slice * 32 + lane;
    float4 wv[U][SK_MR];
    // the first weights before the dependency wait: no kernel writes weights
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < SK_MR; ++r) wv[u][r] = i + u * step < k4 ? __ldg(wr[r] + i + u * step) : zero;
    pdl_wait();
    const float4* xr[N];
#pragma unroll
    for (int n = 0; n < N; ++n) xr[n] = reinterpret_cast<const float4*>(x + (size_t)min(n0 + n, n_rows - 1) * ldx);
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.f;
    while (i < k4) {
        float4 next[U][SK_MR];
        const int j = i + U * step;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < SK_MR; ++r) next[u][r] = j + u * step < k4 ? __ldg(wr[r] + j + u * step) : zero;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = i + u * step < k4;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const float4 xv = in ? xr[n][i + u * step] : zero;
#pragma unroll
                for (int r = 0; r < SK_MR; ++r) {
                    float& a = acc[r * N + n];
                    a = fmaf(xv.x, wv[u][r].x, a);
                    a = fmaf(xv.y, wv[u][r].y, a);
                    a = fmaf(xv.z, wv[u][r].z, a);
                    a = fmaf(xv.w, wv[u][r].w, a);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < SK_MR; ++r) wv[u][r] = next[u][r];
        i = j;
    }
    const float mine = warp_sums<V>(acc);
    if ((lane & ((1 << SHIFT) - 1)) == 0) part[warp][lane >> SHIFT] = mine;
    __syncthreads();
    const int g = threadIdx.x / V, v = threadIdx.x - g * V;
    if (g >= groups) return;
    float sum = 0.f;
    for (int s = 0; s < ks; ++s) sum += part[g * ks + s][v];
    const int m = (blockIdx.x * groups + g) * SK_MR + v / N, n = n0 + v % N;
    if (m >= m_out || n >= n_rows) return;
    const size_t o = (size_t)n * ldo + m;
    out[o] = res ? res[o] + sum : sum;
}

// Many rows: bound by the FMA pipes.  A CTA owns 64 outputs x 64 tokens; groups of 64 threads (8 x 8 numbers a thread: 64 FMA for
// four 16-byte reads of shared memory) take every KS-th k block of 16, each with two buffers of its own, and add their
// sums up in order at the end.  KS is what fills the SMs: 4 groups where one CTA an SM covers the product, 1 where several do.
#define ST_B 64
#define ST_LD 68
#define ST_BUF (2 * SG_BK * ST_LD)          // floats of one buffer: x, then w, [k][row]

template <int KS> constexpr int gemm_tile_smem() { return KS * 2 * ST_BUF * 4; }

template <int KS>
__global__ void __launch_bounds__(64 * KS)
gemm_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, float* out, const float* res, int n_rows, int m_out,
                 int k_in, long long ldx, long long ldw, long long ldo, int wide_out) {
    extern __shared__ __align__(16) float st_smem[];
    pdl_trigger();
    const int group = threadIdx.x / 64, t = threadIdx.x & 63;
    const int tx = t & 7, ty = t >> 3;
    const int m0 = blockIdx.x * ST_B, n0 = blockIdx.y * ST_B;
    float* bufs = st_smem + group * 2 * ST_BUF;
    const int blocks = (k_in + SG_BK - 1) / SG_BK, turns = (blocks + KS - 1) / KS;
    const int lr = t >> 2, lk = (t & 3) * 4;                 // this thread fetches rows lr + 16 i, four numbers from lk on
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 px[4], pw[4];
    auto fetch_w = [&](int turn) {
        const int k = (turn * KS + group) * SG_BK + lk;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = m0 + lr + 16 * i;
            pw[i] = (k < k_in && m < m_out) ? __ldg(reinterpret_cast<const float4*>(w + (size_t)m * ldw + k)) : zero;
        }
    };
    auto fetch_x = [&](int turn) {
        const int k = (turn * KS + group) * SG_BK + lk;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = n0 + lr + 16 * i;
            px[i] = (k < k_in && n < n_rows) ? *reinterpret_cast<const float4*>(x + (size_t)n * ldx + k) : zero;
        }
    };
    auto put = [&](float* buf) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float xv[4] = {px[i].x, px[i].y, px[i].z, px[i].w}, wv[4] = {pw[i].x, pw[i].y, pw[i].z, pw[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                buf[(lk + e) * ST_LD + lr + 16 * i] = xv[e];
                buf[SG_BK * ST_LD + (lk + e) * ST_LD + lr + 16 * i] = wv[e];
            }
        }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    fetch_w(0);
    pdl_wait();
    fetch_x(0);
    put(bufs);
    __syncthreads();
    for (int turn = 0; turn < turns; ++turn) {
        const bool more = turn + 1 < turns;
        if (more) { fetch_w(turn + 1); fetch_x(turn + 1); }
        const float* xs = bufs + (turn & 1) * ST_BUF;
        const float* ws = xs + SG_BK * ST_LD;
#pragma unroll
        for (int kk = 0; kk < SG_BK; ++kk) {
            float xv[8], wv[8];
            *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(xs + kk * ST_LD + ty * 4);
            *reinterpret_cast<float4*>(xv + 4) = *reinterpret_cast<const float4*>(xs + kk * ST_LD + 32 + ty * 4);
            *reinterpret_cast<float4*>(wv) = *reinterpret_cast<const float4*>(ws + kk * ST_LD + tx * 4);
            *reinterpret_cast<float4*>(wv + 4) = *reinterpret_cast<const float4*>(ws + kk * ST_LD + 32 + tx * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        if (more) put(bufs + ((turn + 1) & 1) * ST_BUF);
        __syncthreads();
    }
    if (KS > 1) {                                           // every buffer has been read: the groups' sums meet there
        for (int g = 1; g < KS; ++g) {
            if (group == g) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) st_smem[(i * 8 + j) * 64 + t] = acc[i][j];
            }
            __syncthreads();
            if (group == 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] += st_smem[(i * 8 + j) * 64 + t];
            }
            __syncthreads();
        }
        if (group) return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int n = n0 + (i >> 2) * 32 + ty * 4 + (i & 3);
        if (n >= n_rows) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int m = m0 + half * 32 + tx * 4;
            const size_t o = (size_t)n * ldo + m;
            const float* v = acc[i] + half * 4;
            if (wide_out && m + 3 < m_out) {
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (res) {
                    const float4 old = *reinterpret_cast<const float4*>(res + o);
                    r = make_float4(old.x + r.x, old.y + r.y, old.z + r.z, old.w + r.w);
                }
                *reinterpret_cast<float4*>(out + o) = r;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (m + e < m_out) out[o + e] = res ? res[o + e] + v[e] : v[e];
            }
        }
    }
}

template <int N>
static void launch_few(const float* x, const float* w, float* out, const float* res, int n_rows, int m_out, int k_in,
                       long long ldx, long long ldw, long long ldo, cudaStream_t s) {
    // as many warps share a group of rows as it takes to have some 2,400 warps, down to 32 numbers of k a lane's pass
    const int groups = (m_out + SK_MR - 1) / SK_MR, tokens = (n_rows + N - 1) / N;
    int ks = 1;
    while (ks < SK_WARPS && (long long)groups * tokens * ks < 16 * 148 && k_in / 4 > 32 * ks) ks *= 2;
    const int per = SK_WARPS / ks;
    braid_launch(gemm_few_kernel<N>, dim3((groups + per - 1) / per, tokens), dim3(SK_WARPS * 32), 0, s, x, w, out, res, n_rows, m_out,
                 k_in / 4, ks, ldx, ldw, ldo);
}

template <int KS>
static cudaError_t launch_tile(dim3 grid, const float* x, const float* w, float* out, const float* res, int n_rows, int m_out, int k_in,
                               long long ldx, long long ldw, long long ldo, int wide_out, cudaStream_t s) {
    static bool configured = false;
    if (!configured && gemm_tile_smem<KS>() > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tile_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_tile_smem<KS>());
        if (e != cudaSuccess) return e;
        configured = true;
    }
    return braid_launch(gemm_tile_kernel<KS>, grid, dim3(64 * KS), (size_t)gemm_tile_smem<KS>(), s, x, w, out, res, n_rows, m_out, k_in,
                        ldx, ldw, ldo, wide_out);
}

static int gemm_f32(const float* x, const float* w, float* out, const float* res, int n_rows, int m_out, int k_in, long long ldx,
                    long long ldw, long long ldo, cudaStream_t s) {
    if (n_rows <= SK_MAX_ROWS) {
        if (n_rows == 1) launch_few<1>(x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, s);
        else if (n_rows == 2) launch_few<2>(x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, s);
        else if (n_rows <= 4) launch_few<4>(x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, s);
        else launch_few<8>(x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, s);
        BRAID_LAUNCH_CHECK();
    }
    const dim3 grid((m_out + ST_B - 1) / ST_B, (n_rows + ST_B - 1) / ST_B);
    const long long tiles = (long long)grid.x * grid.y;
    const int wide_out = (ldo % 4 == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)res & 15) == 0) ? 1 : 0;
    cudaError_t e;
    if (tiles <= 148) e = launch_tile<4>(grid, x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, wide_out, s);
    else if (tiles <= 3 * 148) e = launch_tile<2>(grid, x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, wide_out, s);
    else e = launch_tile<1>(grid, x, w, out, res, n_rows, m_out, k_in, ldx, ldw, ldo, wide_out, s);
    if (e != cudaSuccess) { braid_set_error("gemm_simt: %s", cudaGetErrorString(e)); return (int)e; }
    BRAID_LAUNCH_CHECK();
}

extern "C" int braid_gemm_simt(const void* x, const void* w, void* out, const float* res,
                               int in_dtype, int out_dtype, int mode,
                               int n_rows, int m_out, int k_in,
                               long long ldx, long long ldw, long long ldo, void* stream) {
    if (n_rows <= 0 || m_out <= 0) return BRAID_OK;
    if (k_in <= 0) BRAID_REFUSE("gemm_simt: k=%d must be positive", k_in);
    if (mode == 1 && (out_dtype != BRAID_F32 || res == nullptr)) BRAID_REFUSE("gemm_simt: the residual epilogue writes float32 and needs res");
    if (mode != 0 && mode != 1) BRAID_REFUSE("gemm_simt: unknown epilogue %d", mode);
    dim3 grid((m_out + SG_BM - 1) / SG_BM, (n_rows + SG_BN - 1) / SG_BN);
    if (grid.y > 65535) BRAID_REFUSE("gemm_simt: %d rows exceed the grid limit", n_rows);
    cudaStream_t s = (cudaStream_t)stream;
    if (in_dtype == BRAID_F32 && out_dtype == BRAID_F32 && k_in % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 &&
        (((uintptr_t)x | (uintptr_t)w) & 15) == 0)
        return gemm_f32((const float*)x, (const float*)w, (float*)out, mode ? res : nullptr, n_rows, m_out, k_in, ldx, ldw, ldo, s);
#define SG_LAUNCH(T, TO, MODE) braid_launch(gemm_simt_kernel<T, TO, MODE>, dim3(grid), dim3(256), 0, s, (const T*)x, (const T*)w, (TO*)out, res, n_rows, m_out, k_in, ldx, ldw, ldo)
    if (in_dtype == BRAID_F32 && out_dtype == BRAID_F32) { if (mode) SG_LAUNCH(float, float, 1); else SG_LAUNCH(float, float, 0); }
    else if (in_dtype == BRAID_BF16 && out_dtype == BRAID_F32) { if (mode) SG_LAUNCH(__nv_bfloat16, float, 1); else SG_LAUNCH(__nv_bfloat16, float, 0); }
    else if (in_dtype == BRAID_BF16 && out_dtype == BRAID_BF16) SG_LAUNCH(__nv_bfloat16, __nv_bfloat16, 0);
    else BRAID_REFUSE("gemm_simt: unsupported dtype codes in=%d out=%d", in_dtype, out_dtype);
#undef SG_LAUNCH
    BRAID_LAUNCH_CHECK();
}
