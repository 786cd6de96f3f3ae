// What delta.cu and delta_chunk.cu share: the arguments of the gated delta rule (see delta.cu) and its gates.
#pragma once
#include "common.cuh"

#define DELTA_C 64                 // tokens a chunk

struct DeltaArgs {
    const float* q; long long q_stride;          // [rows, groups * dk]
    const float* k; long long k_stride;
    const float* v; long long v_stride;          // [rows, heads * dv]
    const float* z; long long z_stride;          // [rows, heads * dk]: decay logits
    const float* bias;                           // [heads * dk]
    const float* rate;                           // [heads], positive
    const void* b; long long b_stride;           // [rows, heads], run type: the step sizes' logits
    float* out; long long out_stride;            // [rows, heads * dv]
    uint8_t* state; long long state_stride, state_offset;
    const int *q_start, *q_len, *slot_ids;
    int heads, groups, dk, dv;
    int wide_qk, wide_z;                         // rows of q and k, of z start on 16 bytes
    // scratch of the chunked forms: blocks a (chunk, head), see delta_block; the layouts are the forms' own
    float *w, *u, *qd, *kd, *p, *gc, *sc;
    __nv_bfloat16 *wp, *kp;                      // operands in three parts
    int tiles, max_chunks;                       // tiles of value columns
    int settled;                                 // the state may be read before the wait (common.cuh)
};

// The place of chunk c of sequence seq among all chunks of the step: a sequence's chunks lie one after the other, and two
// sequences' never meet (a sequence of n rows takes ceil(n / 64) places, the next one starts at least so many further on).
__device__ __forceinline__ size_t delta_block(const DeltaArgs& a, int seq, int c, int h) {
    return (size_t)(a.q_start[seq] / DELTA_C + seq + c) * a.heads + h;
}

// a decay from its logit: exp(-rate softplus(x))
__device__ __forceinline__ float delta_decay(float x, float rate) {
    return expf(-rate * (fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)))));
}
__device__ __forceinline__ float delta_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ void delta_cp16(uint32_t smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void delta_cp16(void* smem, const void* gmem) { delta_cp16((uint32_t)__cvta_generic_to_shared(smem), gmem); }
__device__ __forceinline__ void delta_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void delta_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The form over chunks for dk <= 128 (delta_chunk.cu): its scratch, and its launches.
long long dlc_floats(long long blocks, int dk, int dv);
int dlc_launch(const DeltaArgs& a, int dtype, int n_seqs, long long blocks, float* work, cudaStream_t s);
