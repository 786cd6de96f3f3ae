// bfloat16 attention of prompts over a latent cache on tcgen05, on expanded keys and values.
//
// The other kernels of latent attention (latent.cu, latent_attn_mma.cu) carry a head's query into the latent space and walk
// the cached rows themselves: 2 (2 kv_rank + rot) FLOPs a query, head and key.  A prompt has many queries for every cached row,
// and there it is cheaper to expand the rows once, key = Wuk c, value = Wuv c for every head (one ordinary product over
// the step's context, 2 kv_rank (dim + vdim) a row and head), and to attend over heads of the ordinary size: 2 (dim + rot +
// vdim) a pair, 640 FLOPs instead of 2,176 for a rank of 512 and heads of 128 + 64.  It also fits tensor memory: the
// 128 x vdim accumulator and two buffers of scores take half of it, where the latent form's 128 x 512 accumulator takes all.
//
//   latent_expand_rows   the context's latents, page after page, from the paged cache into neighbouring rows (the product's
//                        input); rows past a sequence's end become zeros
//   (the product)        [rows, heads x (dim | vdim)] by gemm_tc
//   latent_attn_tc       this file's attention; the rotated key part, one for all heads, is read from the cache
//
// The attention kernel is attn_tc.cu's with one head a CTA: 128 queries of one head, key tiles of one page, warp 0 TMA, warp 1
// MMA, warps 2..5 a softmax row a thread; scores and the accumulator in tensor memory, P back into tensor memory as the
// second product's A operand; two CTAs an SM (one's chain of dependent steps under the other's), which is what sets the
// rings: for heads of 128 two key stages of 24 KB and one value stage.  A score is q_u . k_u + q_r . k_r: the K dimension of the
// first product runs over dim / 64 blocks of the expanded keys and one block with the rotated part (rot <= 64 numbers,
// zeros beyond from TMA's fill).  The output gate, a factor and a sink a head are in the epilogue.
//
// Measured in microseconds (rank 512, heads of 128 + 64 | 128; gathered rows, product and attention together, beside queries into
// the latent space, latent_attn_mma and values out of it): 16 heads, 2,048 tokens 85 beside 725; 512 tokens after 4,096 152
// beside 940 (of which this kernel 99 beside 881); 16 sequences of 20 tokens after 1,024 129 beside 250.  32 heads, two
// sequences of 1,777 and 1,244 tokens: this kernel 85 beside 1,390.
#include "common.cuh"
#include "attn_tc.cuh"
#include "page.h"

#define LA_BM 128
#define LA_BN 64                                 // keys per tile: one page
static_assert(BRAID_PAGE_SIZE == LA_BN, "a key tile of this kernel is one page of 64 positions");
#define LA_THREADS 192
#define LA_QBLOCK_BYTES (128 * 128)              // [128 rows][64 elements] bf16
#define LA_KBLOCK_BYTES (64 * 128)               // [64 positions][64 elements]
#define LA_KST 2
#define LA_BAR_BYTES 192
#define LA_TMEM_COLS 256                         // S0 [0,64) S1 [64,128), O [128, 128 + VDIM)

// Where a sequence's context lies among the step's expanded rows: its pages from the first that any of its queries sees,
// sequence after sequence.  Sequences that bring fewer than min_q tokens have none: their queries stay with the latent form.
// Called by whole warps.
struct LaSpan { int page0, pages, base; };       // first page of the sequence, how many, and the expanded page of the first
__device__ __forceinline__ LaSpan la_span(const int* q_len, const int* kv_before, int seq, int window, int min_q) {
    const int lane = threadIdx.x & 31;
    auto first = [&](int s) { const int lo = window > 0 ? kv_before[s] - window + 1 : 0; return lo > 0 ? lo / LA_BN : 0; };
    auto count = [&](int s) { return q_len[s] >= min_q ? (kv_before[s] + q_len[s] + LA_BN - 1) / LA_BN - first(s) : 0; };
    int n = 0;
    for (int s = lane; s < seq; s += 32) n += count(s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return LaSpan{first(seq), count(seq), n};
}

// ------------------------------------------------------------------ the context's latents in neighbouring rows
struct LaRowsArgs {
    const uint4* cache;          // [pages][64][D]
    uint4* rows;                 // [expanded pages * 64][rank]
    const int *page_table, *q_len, *kv_before;
    int d16, rank16;             // D and rank in runs of 16 bytes
    int table_cols, num_pages, window, min_q, max_pages;
    int* error_flag;
};

__global__ void __launch_bounds__(256)
latent_expand_rows_kernel(LaRowsArgs a) {
    pdl_trigger();
    const int seq = blockIdx.y, p = blockIdx.x;
    const LaSpan at = la_span(a.q_len, a.kv_before, seq, a.window, a.min_q);
    if (p >= at.pages || at.base + p >= a.max_pages) return;
    const int block = at.page0 + p;
    int page = block < a.table_cols ? a.page_table[(size_t)seq * a.table_cols + block] : -1;
    if (page < 0 || page >= a.num_pages) {       // never followed: flagged, page 0 instead
        if (threadIdx.x == 0) atomicExch(a.error_flag, 1);
        page = 0;
    }
    const int live = min(LA_BN, a.kv_before[seq] + a.q_len[seq] - block * LA_BN);
    const uint4* src = a.cache + (size_t)page * LA_BN * a.d16;
    uint4* dst = a.rows + (size_t)(at.base + p) * LA_BN * a.rank16;
    pdl_wait();
#pragma unroll 4
    for (int i = threadIdx.x; i < LA_BN * a.rank16; i += 256) {
        const int r = i / a.rank16, c = i - r * a.rank16;
        dst[i] = r < live ? src[(size_t)r * a.d16 + c] : make_uint4(0, 0, 0, 0);
    }
}

// `max_pages`: expanded pages that `rows` holds; `max_seq_pages`: the most of one sequence.
extern "C" int braid_latent_expand_rows(const void* cache, void* rows, const int* page_table, const int* q_len, const int* kv_before,
                                        int n_seqs, int d, int rank, int table_cols, int num_pages, int window, int min_q, int max_pages,
                                        int max_seq_pages, int* error_flag, void* stream) {
    if (n_seqs <= 0 || max_pages <= 0 || max_seq_pages <= 0) return BRAID_OK;
    if (rank <= 0 || rank % 8 || d % 8 || d < rank || (((uintptr_t)cache | (uintptr_t)rows) & 15)) BRAID_REFUSE("latent_expand_rows: rows of %d numbers, %d of them latent, must be whole runs of 16 bytes", d, rank);
    if (num_pages <= 0 || table_cols <= 0 || n_seqs > 65535) BRAID_REFUSE("latent_expand_rows: %d pages, %d table columns, %d sequences", num_pages, table_cols, n_seqs);
    if (!error_flag) BRAID_REFUSE("latent_expand_rows: error_flag is required");
    LaRowsArgs a{(const uint4*)cache, (uint4*)rows, page_table, q_len, kv_before, d / 8, rank / 8, table_cols, num_pages, window, min_q > 1 ? min_q : 1, max_pages, error_flag};
    braid_launch(latent_expand_rows_kernel, dim3(max_seq_pages, n_seqs), dim3(256), 0, (cudaStream_t)stream, a);
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ attention
struct LatentTcArgs {
    __nv_bfloat16* out;          // [rows, out_row_stride]: head h at column h * VDIM
    const int *page_table, *q_start, *q_len, *kv_before;
    int out_row_stride, heads, table_cols, num_pages, window, min_q, rot, rank;
    float scale_log2, out_scale;
    const float* head_sinks;     // [heads] natural-log scores, or null
    const __nv_bfloat16* head_gate;
    long long gate_stride;
    int* error_flag;
};

template <int DIM, int VDIM>
struct LaSizes {
    static constexpr int KB = DIM / 64 + 1;                    // 64-element blocks of a key: expanded, then the rotated part
    static constexpr int VB = VDIM / 64;
    static constexpr int VST = VDIM == 64 ? 3 : 1;
    static constexpr int Q_BYTES = KB * LA_QBLOCK_BYTES, K_BYTES = KB * LA_KBLOCK_BYTES, V_BYTES = VB * LA_KBLOCK_BYTES;
    static constexpr int SMEM = Q_BYTES + LA_KST * K_BYTES + VST * V_BYTES + LA_BAR_BYTES;
};

template <int DIM, int VDIM>
__global__ void __launch_bounds__(LA_THREADS, 2)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map_qu, const __grid_constant__ CUtensorMap map_qr,
                      const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_kr, LatentTcArgs a) {
    using Z = LaSizes<DIM, VDIM>;
    constexpr int KB = Z::KB, VB = Z::VB, VST = Z::VST;
    pdl_trigger();
    // the swizzled tiles want 1024-byte alignment; two CTAs an SM leave no room for slack, so the start is checked
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(a.error_flag, 1);
        return;
    }
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + Z::Q_BYTES;
    uint8_t* sV = sK + LA_KST * Z::K_BYTES;
    uint64_t* bars = (uint64_t*)(sV + VST * Z::V_BYTES);
    uint64_t* q_full = bars;
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + LA_KST;
    uint64_t* v_full = k_empty + LA_KST;
    uint64_t* v_empty = v_full + VST;
    uint64_t* s_full = v_empty + VST;              // [2]
    uint64_t* p_ready = s_full + 2;                // [2], in turn (see attn_tc.cu)
    uint64_t* pv_done = p_ready + 2;
    uint32_t* tmem_slot = (uint32_t*)(pv_done + 1);
    static_assert((1 + 2 * LA_KST + 2 * VST + 5) * 8 + 8 <= LA_BAR_BYTES, "the barriers outgrow their bytes");
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // late tokens see the most keys: their CTAs start first
    const int head = blockIdx.x, seq = blockIdx.y, tile = gridDim.z - 1 - blockIdx.z;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < LA_KST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
        for (int s = 0; s < VST; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1);
        mbar_init(&p_ready[0], 128); mbar_init(&p_ready[1], 128); mbar_init(pv_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, LA_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_o = tmem_base + 128;
    pdl_wait();

    const LaSpan span = la_span(a.q_len, a.kv_before, seq, a.window, a.min_q);
    const int q_len = a.q_len[seq];
    const int tok0 = tile * LA_BM;
    const bool active = tok0 < q_len && q_len >= a.min_q;      // uniform over the CTA
    const int q_start = a.q_start[seq], kv_before = a.kv_before[seq];
    const int n_tok = active ? min(LA_BM, q_len - tok0) : 0;
    const int pos_min = kv_before + tok0, pos_max = pos_min + n_tok - 1;
    const int k_lo = (a.window > 0 && pos_min - a.window + 1 > 0) ? pos_min - a.window + 1 : 0;
    const int t_lo = k_lo / LA_BN, t_hi = active ? pos_max / LA_BN + 1 : 0;
    const int n_tiles = active ? t_hi - t_lo : 0;

    if (warp == 0) {
        if (lane == 0 && active) {
            mbar_expect_tx(q_full, (uint32_t)Z::Q_BYTES);
#pragma unroll
            for (int b = 0; b < KB - 1; ++b) tma_load_3d(&map_qu, q_full, sQ + b * LA_QBLOCK_BYTES, b * 64, head, q_start + tok0);
            tma_load_3d(&map_qr, q_full, sQ + (KB - 1) * LA_QBLOCK_BYTES, a.rank, head, q_start + tok0);
            const int* table = a.page_table + (size_t)seq * a.table_cols;
            const int v_col = a.heads * DIM + head * VDIM;
            // key and value tiles go out independently, each as soon as its stage is free
            int jk = 0, jv = 0;
            uint32_t idle = 0;
            uint64_t idle_since = 0;
            while (jk < n_tiles || jv < n_tiles) {
                const bool k_turn = jk < n_tiles && mbar_try_wait(&k_empty[jk % LA_KST], (uint32_t)((jk / LA_KST) & 1) ^ 1u);
                const bool v_turn = !k_turn && jv < n_tiles && mbar_try_wait(&v_empty[jv % VST], (uint32_t)((jv / VST) & 1) ^ 1u);
                if (k_turn) {
                    int page = (t_lo + jk < a.table_cols) ? table[t_lo + jk] : -1;
                    if (page < 0 || page >= a.num_pages) {          // a visible position without a page: the table is broken
                        atomicExch(a.error_flag, 1);
                        page = 0;
                    }
                    const int st = jk % LA_KST, row = (span.base + t_lo - span.page0 + jk) * LA_BN;
                    uint8_t* dst = sK + st * Z::K_BYTES;
                    mbar_expect_tx(&k_full[st], Z::K_BYTES);
#pragma unroll
                    for (int b = 0; b < KB - 1; ++b) tma_load_2d(&map_kv, &k_full[st], dst + b * LA_KBLOCK_BYTES, head * DIM + b * 64, row);
                    tma_load_2d(&map_kr, &k_full[st], dst + (KB - 1) * LA_KBLOCK_BYTES, a.rank, page * LA_BN);
                    ++jk;
                } else if (v_turn) {
                    const int st = jv % VST, row = (span.base + t_lo - span.page0 + jv) * LA_BN;
                    mbar_expect_tx(&v_full[st], Z::V_BYTES);
#pragma unroll
                    for (int b = 0; b < VB; ++b) tma_load_2d(&map_kv, &v_full[st], sV + st * Z::V_BYTES + b * LA_KBLOCK_BYTES, v_col + b * 64, row);
                    ++jv;
                }
                if (k_turn || v_turn) { idle = 0; idle_since = 0; continue; }
                if (++idle >= TC_SPIN_LIMIT) { *abort_flag = 1; break; }
                if ((idle & 1023u) == 1023u) {              // the same bound as mbar_wait: time on the device's clock
                    if (*abort_flag) break;
                    const uint64_t now = global_timer_ns();
                    if (idle_since == 0) idle_since = now;
                    else if (now - idle_since > TC_WAIT_LIMIT_NS) { *abort_flag = 1; break; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && active) {
            constexpr uint32_t idesc_qk = umma_idesc_bf16(LA_BM, LA_BN);
            constexpr uint32_t idesc_pv = umma_idesc_bf16_b_mn(LA_BM, VDIM);
            bool ok = mbar_wait(q_full, 0, abort_flag);
            const uint64_t dq = umma_desc_sw128(smem_u32(sQ));
            const uint64_t dk = umma_desc_sw128(smem_u32(sK));
            const uint64_t dv = umma_desc_sw128_mn(smem_u32(sV), LA_KBLOCK_BYTES);
            const uint32_t q_lo = (uint32_t)dq, k_lo32 = (uint32_t)dk, v_lo = (uint32_t)dv;
            const uint32_t kq_hi = (uint32_t)(dq >> 32), v_hi = (uint32_t)(dv >> 32);
            const int rot_steps = a.rot / 16;
            auto issue_pv = [&](int i, int st) -> bool {
                if (!mbar_wait(&v_full[st], (uint32_t)((i / VST) & 1), abort_flag)) return false;
                if (!mbar_wait(&p_ready[i & 1], (uint32_t)((i >> 1) & 1), abort_flag)) return false;     // P written, O rescaled
                tc_fence_after();
                const uint32_t vs_lo = v_lo + (uint32_t)((st * Z::V_BYTES) >> 4);
                const uint32_t tp = tmem_base + (i & 1) * LA_BN;
                umma_ts_lohi(tmem_o, tp, vs_lo, v_hi, idesc_pv, i > 0 ? 1u : 0u);
#pragma unroll
                for (int ks = 1; ks < LA_BN / 16; ++ks)
                    umma_ts_lohi(tmem_o, tp + ks * 8, vs_lo + (uint32_t)((ks * 16 * 128) >> 4), v_hi, idesc_pv, 1u);
                umma_commit(pv_done);
                umma_commit(&v_empty[st]);
                return true;
            };
            int kst = 0, vst = 0;                  // ring stages of key tile j and of value tile j - 1
            for (int j = 0; j < n_tiles && ok; ++j) {
                ok = mbar_wait(&k_full[kst], (uint32_t)((j / LA_KST) & 1), abort_flag);
                // S of tile j goes where S and P of tile j - 2 were: the second product of tile j - 2 has to be complete
                if (ok && j >= 2) ok = mbar_wait(pv_done, (uint32_t)(j & 1), abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ks_lo = k_lo32 + (uint32_t)((kst * Z::K_BYTES) >> 4);
                const uint32_t ts = tmem_base + (j & 1) * LA_BN;
#pragma unroll
                for (int ks = 0; ks < DIM / 16; ++ks) {
                    const uint32_t qoff = ((ks >> 2) * LA_QBLOCK_BYTES + (ks & 3) * 32) >> 4, koff = ((ks >> 2) * LA_KBLOCK_BYTES + (ks & 3) * 32) >> 4;
                    umma_ss_lohi(ts, q_lo + qoff, kq_hi, ks_lo + koff, kq_hi, idesc_qk, ks > 0 ? 1u : 0u);
                }
                for (int ks = 0; ks < rot_steps; ++ks)
                    umma_ss_lohi(ts, q_lo + (((KB - 1) * LA_QBLOCK_BYTES + ks * 32) >> 4), kq_hi, ks_lo + (((KB - 1) * LA_KBLOCK_BYTES + ks * 32) >> 4),
                                 kq_hi, idesc_qk, 1u);
                umma_commit(&s_full[j & 1]);
                umma_commit(&k_empty[kst]);
                if (++kst == LA_KST) kst = 0;
                if (j > 0) {
                    ok = issue_pv(j - 1, vst);
                    if (++vst == VST) vst = 0;
                }
            }
            if (ok && n_tiles > 0) issue_pv(n_tiles - 1, vst);
        }
    } else if (active) {
        const int quarter = warp & 3;                          // tensor-memory lanes 32 * quarter ...
        const int tl = quarter * 32 + lane;                    // this thread's row: a token
        const bool valid = tl < n_tok;
        const int pos = valid ? pos_min + tl : -1;
        const int lo = (a.window > 0) ? pos - a.window + 1 : 0;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        float m = -INFINITY, l = 0.f;
        const float sc = a.scale_log2;
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int st = j & 1;
            ok = mbar_wait(&s_full[st], (uint32_t)((j >> 1) & 1), abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            float sv[64];
            tmem_ld32x2(tmem_base + st * LA_BN + lane_addr, sv);
            const int key0 = (t_lo + j) * LA_BN;
            const bool all_visible = (key0 + LA_BN - 1 <= pos_min) && (a.window == 0 || key0 >= pos_max - a.window + 1);
            float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
            if (!all_visible) {
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    const int key = key0 + i;
                    if (!(key <= pos && key >= lo)) sv[i] = -INFINITY;
                }
            }
            if (valid || !all_visible) {
#pragma unroll
                for (int i = 0; i < 64; i += 4) {
                    mx0 = fmaxf(mx0, sv[i]); mx1 = fmaxf(mx1, sv[i + 1]);
                    mx2 = fmaxf(mx2, sv[i + 2]); mx3 = fmaxf(mx3, sv[i + 3]);
                }
            }
            const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * sc;   // scale > 0 commutes with the maximum
            // raise m only when the tile towers over it; -inf + 8 = -inf, so the first finite maximum always does
            const bool raise = mx > m + FA_RAISE;
            const float factor = raise ? exp2f(m - mx) : 1.f;                     // exp2(-inf) = 0: nothing was summed yet
            if (raise) m = mx;
            // a row that is no query (past the tile's tokens) sums nothing: exp2(-inf) = 0
            const float ms = (!valid && all_visible) ? INFINITY : ((m == -INFINITY) ? 0.f : m);
            float sum0 = 0.f, sum1 = 0.f;
            uint32_t pk[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float p0 = exp2f(fmaf(sv[2 * i], sc, -ms));
                const float p1 = exp2f(fmaf(sv[2 * i + 1], sc, -ms));
                sum0 += p0;
                sum1 += p1;
                __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
                pk[i] = *reinterpret_cast<uint32_t*>(&b);
            }
            l = l * factor + (sum0 + sum1);
            tmem_st32_nowait(tmem_base + st * LA_BN + lane_addr, pk);      // over the first half of this row's scores
            if (j > 0) {
                // looked at every tile: a parity wait only tells apart a barrier that is at most one phase off
                ok = mbar_wait(pv_done, (uint32_t)((j - 1) & 1), abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (__any_sync(0xffffffffu, raise)) {          // tensor-memory loads and stores take the whole warp
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < VB; ++h) {
                        float ov[64];
                        tmem_ld32x2(tmem_o + h * 64 + lane_addr, ov);
#pragma unroll
                        for (int i = 0; i < 64; ++i) ov[i] *= factor;
                        tmem_st32x2(tmem_o + h * 64 + lane_addr, ov);
                    }
                }
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&p_ready[st]);
        }
        if (ok && n_tiles > 0) {
            ok = mbar_wait(pv_done, (uint32_t)((n_tiles - 1) & 1), abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                tc_fence_after();
                // the sink joins the sum where the row is finished: l counts in units of 2^m
                float inv = a.out_scale / (a.head_sinks ? l + exp2f(a.head_sinks[head] * 1.4426950408889634f - m) : l);
                const size_t row = (size_t)(q_start + tok0 + tl);
                if (a.head_gate && valid) inv *= 1.f / (1.f + expf(-__bfloat162float(a.head_gate[row * a.gate_stride + head])));
                __nv_bfloat16* dst = a.out + row * a.out_row_stride + (size_t)head * VDIM;
#pragma unroll
                for (int h = 0; h < VB; ++h) {
                    float ov[64];
                    tmem_ld32x2(tmem_o + h * 64 + lane_addr, ov);
                    if (valid) {
#pragma unroll
                        for (int c = 0; c < 64; c += 8) {
                            uint32_t w[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                __nv_bfloat162 b = __floats2bfloat162_rn(ov[c + 2 * i] * inv, ov[c + 2 * i + 1] * inv);
                                w[i] = *reinterpret_cast<uint32_t*>(&b);
                            }
                            *reinterpret_cast<uint4*>(dst + h * 64 + c) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicExch(a.error_flag, 1);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, LA_TMEM_COLS);
    }
}

static int la_map(CUtensorMap* map, int dims_n, const void* base, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    TcEncodeTiledFn fn = tc_encode_tiled_fn();
    if (!fn) BRAID_REFUSE("latent_attn_tc: the driver does not export cuTensorMapEncodeTiled");
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, dims_n, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) BRAID_REFUSE("latent_attn_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
    return BRAID_OK;
}

template <int DIM, int VDIM>
static int launch_latent_tc(const CUtensorMap& qu, const CUtensorMap& qr, const CUtensorMap& kv, const CUtensorMap& kr, const LatentTcArgs& a,
                            dim3 grid, cudaStream_t s) {
    constexpr int SMEM = LaSizes<DIM, VDIM>::SMEM;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(latent_attn_tc_kernel<DIM, VDIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) { braid_set_error("latent_attn_tc: cannot reserve %d bytes of shared memory: %s", SMEM, cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    braid_launch(latent_attn_tc_kernel<DIM, VDIM>, grid, dim3(LA_THREADS), (size_t)SMEM, s, qu, qr, kv, kr, a);
    BRAID_LAUNCH_CHECK();
}

extern "C" int braid_latent_attn_tc_supported(int dim, int rot, int vdim, int rank) {
    return ((dim == 128 && vdim == 128) || (dim == 64 && vdim == 64)) && rot > 0 && rot <= 64 && rot % 16 == 0 && rank > 0 && rank % 8 == 0;
}

// q_u [rows, heads, dim] (a view: `qu_head` elements from head to head, `qu_row` from row to row), q_lat [rows, heads, rank + rot]
// with the rotated parts from column `rank` on; kv [kv_rows, heads * (dim + vdim)] the expanded keys, then values; cache
// [num_pages][64][rank + rot].
extern "C" int braid_latent_attn_tc(const void* q_u, long long qu_head, long long qu_row, const void* q_lat, const void* kv, long long kv_rows,
                                    const void* cache, int num_pages, void* out, const int* page_table, const int* q_start,
                                    const int* q_len, const int* kv_before, int rows, int n_seqs, int max_q_len, int heads, int dim,
                                    int rot, int vdim, int rank, int table_cols, int window, int min_q, int out_row_stride, float scale,
                                    float out_scale, const float* head_sinks, const void* head_gate, long long gate_stride,
                                    int* error_flag, void* stream) {
    if (rows <= 0 || n_seqs <= 0 || max_q_len <= 0) return BRAID_OK;
    if (!braid_latent_attn_tc_supported(dim, rot, vdim, rank)) BRAID_REFUSE("latent_attn_tc: not built for heads of %d + %d, values of %d, rank %d", dim, rot, vdim, rank);
    if (heads <= 0 || num_pages <= 0 || table_cols <= 0 || kv_rows <= 0) BRAID_REFUSE("latent_attn_tc: %d heads, %d pages, %d table columns", heads, num_pages, table_cols);
    if ((((uintptr_t)q_u | (uintptr_t)q_lat | (uintptr_t)kv | (uintptr_t)cache | (uintptr_t)out) & 15) || qu_head % 8 || qu_row % 8 || out_row_stride % 8)
        BRAID_REFUSE("latent_attn_tc: operands and their rows must start on 16 bytes");
    if (!error_flag) BRAID_REFUSE("latent_attn_tc: error_flag is required");
    // the maximum is taken, and keys are masked, before the factor
    if (!(scale > 0.f)) BRAID_REFUSE("latent_attn_tc: the factor on the scores must be positive, not %g", (double)scale);
    const int D = rank + rot;
    const cuuint64_t wide = (cuuint64_t)heads * (dim + vdim);
    CUtensorMap mqu, mqr, mkv, mkr;
    const cuuint32_t qbox[3] = {64, 1, LA_BM}, kbox[2] = {64, LA_BN};
    {
        const cuuint64_t dims[3] = {(cuuint64_t)dim, (cuuint64_t)heads, (cuuint64_t)rows}, st[2] = {(cuuint64_t)qu_head * 2, (cuuint64_t)qu_row * 2};
        if (int rc = la_map(&mqu, 3, q_u, dims, st, qbox)) return rc;
    }
    {
        const cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)heads, (cuuint64_t)rows}, st[2] = {(cuuint64_t)D * 2, (cuuint64_t)heads * D * 2};
        if (int rc = la_map(&mqr, 3, q_lat, dims, st, qbox)) return rc;
    }
    {
        const cuuint64_t dims[2] = {wide, (cuuint64_t)kv_rows}, st[1] = {wide * 2};
        if (int rc = la_map(&mkv, 2, kv, dims, st, kbox)) return rc;
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)num_pages * LA_BN}, st[1] = {(cuuint64_t)D * 2};
        if (int rc = la_map(&mkr, 2, cache, dims, st, kbox)) return rc;
    }
    const long long tiles = (max_q_len + LA_BM - 1) / LA_BM;
    if (tiles > 65535 || n_seqs > 65535) BRAID_REFUSE("latent_attn_tc: the step exceeds the grid limits (%lld token tiles, %d sequences)", tiles, n_seqs);
    LatentTcArgs a{(__nv_bfloat16*)out, page_table, q_start, q_len, kv_before, out_row_stride, heads, table_cols, num_pages, window, min_q > 1 ? min_q : 1, rot, rank,
                   scale * 1.4426950408889634f, out_scale, head_sinks, (const __nv_bfloat16*)head_gate, gate_stride, error_flag};
    const dim3 grid(heads, n_seqs, (unsigned)tiles);
    cudaStream_t s = (cudaStream_t)stream;
    if (dim == 128) return launch_latent_tc<128, 128>(mqu, mqr, mkv, mkr, a, grid, s);
    return launch_latent_tc<64, 64>(mqu, mqr, mkv, mkr, a, grid, s);
}
