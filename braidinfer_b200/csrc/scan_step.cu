// The linear recurrence of scan.cu for steps of one token a sequence:  S <- diag(a) S + (kappa k) v^T,  o = S^T (q_scale q) + skip v,
// and, where a CTA holds all the columns of a norm's group, the gated norm of o (gated_norm.cuh) in the same kernel.
//
// Such a step is a read and a write of the state and otherwise latency.  A CTA owns (head, sequence, COLS value columns); eight row groups
// of threads take every eighth key row, four neighbouring columns a thread, so that a warp moves whole rows 16 bytes a lane.  The
// state is asked for before the wait for the kernel's predecessor where that is safe (`settled`, common.cuh), all of it at once; what comes from
// the projections is one trip after it.  The walk over several tokens (linear_scan_kernel) stages eight tokens whatever there are, moves the
// state four bytes a lane and is several times the code, which every SM fetches anew between two kernels.  Between the other kernels of a
// decode step, walk / this, us: constant decays, 4 sequences of 8 heads of 128 x 256 14.5 / 3.2; a decay a head, 8 sequences of 32 heads of
// 64 x 64 8.5 / 2.4; a decay a channel, 8 sequences of 4 heads of 64 x 128, with the norm's kernel 7.2 / 3.3.
#include "common.cuh"
#include "gated_norm.cuh"

#define STEP_RG 8                          // row groups
#define STEP_CHANNEL 0                     // the modes of scan.cu
#define STEP_HEAD 1
#define STEP_CONST 3

struct ScanStepArgs {
    const void *q, *k, *v;
    long long q_stride, k_stride, v_stride;
    const void* gate; long long gate_stride;   // channel: float32 logits; head: run type; constant: float32 [heads]
    const void *gate_bias, *a_log, *skip;      // run type
    float* out; long long out_stride;          // null where the norm is done here
    uint8_t* state; long long state_stride, state_offset;
    const int *q_start, *q_len, *slot_ids;
    int heads, groups, dv, act_silu;
    float q_scale, inv_tau;
    // gated norm over the head's columns: y = o / rms(o) * w * act(z) * out_scale
    const void* z; long long z_stride;
    const void* w; void* y; long long y_stride;
    int gate_sigmoid;
    float eps, out_scale;
    int settled;                               // the state may be read before the wait (common.cuh)
};

// four neighbouring numbers
__device__ __forceinline__ void step_load4(const float* p, float* v) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void step_load4(const __nv_bfloat16* p, float* v) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u);
    v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
}
__device__ __forceinline__ void step_store4(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void step_store4(__nv_bfloat16* p, const float* v) {
    const __nv_bfloat162 x = __floats2bfloat162_rn(v[0], v[1]), y = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
}

template <typename T, int MODE, int DK, int COLS>
__global__ void __launch_bounds__(STEP_RG * COLS / 4)
scan_step_kernel(const __grid_constant__ ScanStepArgs a) {
    constexpr int CG = COLS / 4, NT = STEP_RG * CG, R = DK / STEP_RG;
    __shared__ float sq[DK], sk[DK], sa[MODE == STEP_CHANNEL ? DK : 1];
    __shared__ float4 part[STEP_RG][CG];
    __shared__ float red[32];
    pdl_trigger();
    const int h = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x, cg = tid % CG, rg = tid / CG, col = blockIdx.z * COLS + cg * 4;
    if (a.q_len[seq] <= 0) return;
    const size_t row = a.q_start[seq];
    const int g = h / (a.heads / a.groups);
    float4* S = (float4*)((float*)(a.state + (size_t)a.slot_ids[seq] * a.state_stride + a.state_offset) + (size_t)h * DK * a.dv + (size_t)rg * a.dv + col);
    const size_t step = (size_t)STEP_RG * a.dv / 4;
    if (!a.settled) pdl_wait();
    float4 s[R];
#pragma unroll
    for (int j = 0; j < R; ++j) s[j] = S[j * step];
    float ah = 1.f, kap = 1.f, skip = 0.f, bias = 0.f;
    if (MODE == STEP_HEAD) {
        ah = -expf(to_f32(((const T*)a.a_log)[h]));
        bias = to_f32(((const T*)a.gate_bias)[h]);
        if (a.skip) skip = to_f32(((const T*)a.skip)[h]);
    }
    if (MODE == STEP_CONST) ah = ((const float*)a.gate)[h];
    const bool silu = MODE == STEP_CONST && a.act_silu;
    auto staged = [&](float x) { return silu ? (sizeof(T) == 2 ? glu_act_fast(x, BRAID_ACT_SILU) : silu_f32(x)) : x; };
    pdl_wait();
    float vv[4], zz[4];
    step_load4((const T*)a.v + row * a.v_stride + (size_t)h * a.dv + col, vv);
    if (a.y && rg == 0) step_load4((const T*)a.z + row * a.z_stride + (size_t)h * a.dv + col, zz);
    if (MODE == STEP_HEAD) {
        const float x = to_f32(((const T*)a.gate)[row * a.gate_stride + h]) + bias;
        kap = x > 20.f ? x : log1pf(expf(x));
        ah = expf(ah * kap);
    }
    for (int i = tid; i < DK; i += NT) {
        sq[i] = staged(to_f32(((const T*)a.q)[row * a.q_stride + (size_t)g * DK + i])) * a.q_scale;
        sk[i] = staged(to_f32(((const T*)a.k)[row * a.k_stride + (size_t)g * DK + i])) * (MODE == STEP_HEAD ? kap : 1.f);
        if (MODE == STEP_CHANNEL) {
            const float x = ((const float*)a.gate)[row * a.gate_stride + (size_t)h * DK + i] + to_f32(((const T*)a.gate_bias)[(size_t)h * DK + i]);
            sa[i] = expf((fminf(x, 0.f) - log1pf(expf(-fabsf(x)))) * a.inv_tau);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) vv[e] = staged(vv[e]);
    __syncthreads();
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = rg + j * STEP_RG;
        const float kk = sk[i], qq = sq[i], av = MODE == STEP_CHANNEL ? sa[i] : ah;
        s[j].x = fmaf(av, s[j].x, kk * vv[0]);
        s[j].y = fmaf(av, s[j].y, kk * vv[1]);
        s[j].z = fmaf(av, s[j].z, kk * vv[2]);
        s[j].w = fmaf(av, s[j].w, kk * vv[3]);
        o.x = fmaf(s[j].x, qq, o.x);
        o.y = fmaf(s[j].y, qq, o.y);
        o.z = fmaf(s[j].z, qq, o.z);
        o.w = fmaf(s[j].w, qq, o.w);
    }
    part[rg][cg] = o;
    __syncthreads();
    if (rg == 0) {
        float t[4] = {skip * vv[0], skip * vv[1], skip * vv[2], skip * vv[3]};
#pragma unroll
        for (int r = 0; r < STEP_RG; ++r) {
            const float4 x = part[r][cg];
            t[0] += x.x; t[1] += x.y; t[2] += x.z; t[3] += x.w;
        }
        o = make_float4(t[0], t[1], t[2], t[3]);
        if (!a.y) step_store4(a.out + row * a.out_stride + (size_t)h * a.dv + col, t);
    }
    if (a.y) {
        const float ss = block_sum(rg == 0 ? o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w : 0.f, red);
        if (rg == 0) {
            const float r = 1.f / sqrtf(ss / (float)COLS + a.eps), u[4] = {o.x, o.y, o.z, o.w};
            float wv[4], t[4];
            step_load4((const T*)a.w + cg * 4, wv);
#pragma unroll
            for (int e = 0; e < 4; ++e) t[e] = u[e] * r * wv[e] * norm_gate(zz[e], a.gate_sigmoid) * a.out_scale;
            step_store4((T*)a.y + row * a.y_stride + (size_t)h * a.dv + col, t);
        }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) S[j * step] = s[j];
}

template <typename T, int DK, int COLS>
static void launch_scan_step(const ScanStepArgs& a, int mode, int n_seqs, cudaStream_t s) {
    const dim3 grid(a.heads, n_seqs, a.dv / COLS), block(STEP_RG * COLS / 4);
    if (mode == STEP_CHANNEL) braid_launch(scan_step_kernel<T, STEP_CHANNEL, DK, COLS>, grid, block, 0, s, a);
    else if (mode == STEP_HEAD) braid_launch(scan_step_kernel<T, STEP_HEAD, DK, COLS>, grid, block, 0, s, a);
    else braid_launch(scan_step_kernel<T, STEP_CONST, DK, COLS>, grid, block, 0, s, a);
}
template <typename T, int DK>
static int launch_scan_step_cols(const ScanStepArgs& a, int mode, int n_seqs, cudaStream_t s) {
    // with a norm to do, a CTA a head; else CTAs of 64 columns
    if (!a.y || a.dv == 64) launch_scan_step<T, DK, 64>(a, mode, n_seqs, s);
    else if (a.dv == 128) launch_scan_step<T, DK, 128>(a, mode, n_seqs, s);
    else launch_scan_step<T, DK, 256>(a, mode, n_seqs, s);
    BRAID_LAUNCH_CHECK();
}

// One token a sequence (q_len 0 or 1).  dk 64 or 128, dv a multiple of 64; v, state and results on 16 bytes (8 for bfloat16 rows).  With y:
// out is not written, y = the gated norm of every head's columns, dv 64, 128 or 256.
extern "C" int braid_scan_step(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                               const void* gate, long long gate_stride, const void* gate_bias, const void* a_log, const void* skip,
                               float* out, long long out_stride, void* state, long long state_stride, long long state_offset,
                               const int* q_start, const int* q_len, const int* slot_ids, int dtype, int mode, int n_seqs, int heads,
                               int groups, int dk, int dv, float q_scale, float inv_tau, int act_silu, const void* z, long long z_stride,
                               const void* w, void* y, long long y_stride, int gate_sigmoid, float eps, float out_scale, int settled,
                               void* stream) {
    if (n_seqs <= 0) return BRAID_OK;
    if (heads <= 0 || groups <= 0 || heads % groups) BRAID_REFUSE("scan_step: %d heads do not divide into %d groups", heads, groups);
    if ((dk != 64 && dk != 128) || dv <= 0 || dv % 64) BRAID_REFUSE("scan_step: built for keys of 64 or 128 and values in multiples of 64, not %d x %d", dk, dv);
    if (mode != STEP_CHANNEL && mode != STEP_HEAD && mode != STEP_CONST) BRAID_REFUSE("scan_step: unknown decay mode %d", mode);
    if (act_silu && mode != STEP_CONST) BRAID_REFUSE("scan_step: silu on what is given goes with a constant decay a head");
    if (dtype != BRAID_F32 && dtype != BRAID_BF16) BRAID_REFUSE("scan_step: unknown dtype code %d", dtype);
    if (!state || (((uintptr_t)state | (uintptr_t)state_offset | (uintptr_t)state_stride) & 15)) BRAID_REFUSE("scan_step: the state must start on 16 bytes");
    const uintptr_t rows = dtype == BRAID_F32 ? 15 : 7;
    if (((uintptr_t)v & rows) || v_stride % 4) BRAID_REFUSE("scan_step: rows of v must start on %d bytes", (int)rows + 1);
    if (!y && (!out || ((uintptr_t)out & 15) || out_stride % 4)) BRAID_REFUSE("scan_step: results must start on 16 bytes");
    if (y && ((dv != 64 && dv != 128 && dv != 256) || !z || !w || (((uintptr_t)z | (uintptr_t)w | (uintptr_t)y) & rows) || z_stride % 4 || y_stride % 4))
        BRAID_REFUSE("scan_step: the norm is done for heads of 64, 128 or 256 columns whose rows allow moves of four numbers, not %d", dv);
    if (n_seqs > 65535 || dv / 64 > 65535) BRAID_REFUSE("scan_step: the step exceeds the grid limits");
    ScanStepArgs a{q, k, v, q_stride, k_stride, v_stride, gate, gate_stride, gate_bias, a_log, skip, out, out_stride, (uint8_t*)state,
                   state_stride, state_offset, q_start, q_len, slot_ids, heads, groups, dv, act_silu, q_scale, inv_tau, z, z_stride, w, y,
                   y_stride, gate_sigmoid, eps, out_scale, settled};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == BRAID_F32) return dk == 64 ? launch_scan_step_cols<float, 64>(a, mode, n_seqs, s) : launch_scan_step_cols<float, 128>(a, mode, n_seqs, s);
    return dk == 64 ? launch_scan_step_cols<__nv_bfloat16, 64>(a, mode, n_seqs, s) : launch_scan_step_cols<__nv_bfloat16, 128>(a, mode, n_seqs, s);
}
