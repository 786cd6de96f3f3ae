// The experts' products of prompts on pairs of SMs (tcgen05.mma.cta_group::2), bfloat16, float32 accumulation in tensor memory:
//   out[slot, m] = sum_k x[slot, k] * w[expert of the slot, m, k]
// for slots sorted by expert (moe.cu, moe_plan with tiles of MT_CHUNK slots).  The product itself is gemm_tc2.cu's: two CTAs compute
// one [256 weight rows x up to 256 slots] tile, each loading its own half of both operands, six stages of 32 KB.  What
// differs:
//   - a tile belongs to one expert: its weight rows start at the expert's first row of the stack, its slots are the
//     expert's own (a "wide tile" of the plan: up to eight chunks of 32 slots, an expert's chunks shared out evenly), and the
//     MMA is as wide as they are (N = 32 a chunk);
//   - how many tiles there are is known on the device only (the plan's meta), so the grid is one pair an SM pair and the
//     walk ends where the plan says;
//   - units run expert by expert, weight tile by weight tile, an expert's wide tiles innermost, so that neighbouring pairs
//     share a weight tile and every weight comes from memory once.
// The slots' rows lie one after the other (moe_gather_kernel copies the tokens' rows there): a TMA box holds neighbouring rows.
//
// Bound by the weights' bytes where an expert sees up to some 200 tokens, by the tensor cores and power beyond.  Measured in
// microseconds, plan, gathered rows, gate+up and down together, beside the better of the mma.sync kernels of moe.cu (tiles of 16 or
// 64 slots), L2 flushed; in brackets what the weights in use or the products take at 6.55 TB/s and 1.65 PFLOP/s:
//   64 experts of 2048 x 1408, 6 a token: 8 tokens 139 beside 157 (100), 256 tokens 213 beside 280 (169), 2,048 tokens
//   255 beside 894 (169), 4,096 tokens 435 beside 1,668 (258)
//   8 experts of 4096 x 7168, 2 a token: 1 token 111 beside 184 (54), 8 tokens 256 beside 293 (215), 2,048 tokens 642 beside 2,625 (437)
//   16 experts of 1024 x 1024, 2 a token: 1 token 32 beside 39, 2,048 tokens 68 beside 133 (16)
#include "common.cuh"
#include "tcgen05_pair.cuh"

#define MT_BLOCK_M 128          // weight rows of one CTA (256 a pair)
#define MT_BLOCK_K 64
#define MT_UMMA_K 16
#define MT_STAGES 6
#define MT_THREADS 192
#define MT_A_BYTES (MT_BLOCK_M * MT_BLOCK_K * 2)
#define MT_B_BYTES (128 * MT_BLOCK_K * 2)
#define MT_STAGE_BYTES (MT_A_BYTES + MT_B_BYTES)
#define MT_CHUNK 32              // slots of a plan tile, of a tensor-memory load and of a staging tile
#define MT_OUT_BYTES (MT_CHUNK * MT_BLOCK_M * 2)          // one staging tile: [32 slots][128 outputs] bfloat16
#define MT_SMEM_BYTES (MT_STAGES * MT_STAGE_BYTES + 2 * MT_OUT_BYTES + 1024 + 256)
#define MT_TMEM_COLS 512

struct MoeTcArgs {
    const int* tile_expert;    // expert of every plan tile of MT_CHUNK slots
    const int4* wide;          // wide tiles: first slot, chunks, first wide tile of the expert, the expert's wide tiles
    const int* meta;           // [1]: wide tiles in use
    const int* slot_pair;
    const float* in_wgt;       // gated: a weight a pair on the expert's input, or null
    int m_tiles, w_rows, total_kb;     // tiles of 256 weight rows and rows an expert, k blocks of 64
    int m_out, max_wide;
    int* error_flag;
};

struct MtUnit { int m0, slot0, chunks, expert; };

struct MtWalk {
    const MoeTcArgs& a;
    int u, n;
    __device__ MtWalk(const MoeTcArgs& a_) : a(a_) {
        u = blockIdx.x / 2;
        const int wide = a.meta[1];
        n = (wide < a.max_wide ? wide : a.max_wide) * a.m_tiles;
    }
    __device__ bool next(MtUnit& t) {
        if (u >= n) return false;
        const int4 any = a.wide[u / a.m_tiles];                          // a wide tile of this unit's expert
        const int r = u - any.z * a.m_tiles, mt = r / any.w;
        const int4 own = a.wide[any.z + (r - mt * any.w)];
        t.m0 = mt * 2 * MT_BLOCK_M;
        t.slot0 = own.x;
        t.chunks = own.y;
        t.expert = a.tile_expert[own.x / MT_CHUNK];
        u += gridDim.x / 2;
        return true;
    }
};

// MODE 0: out = product; 1: gate and up rows interleaved in blocks of 16, out = silu(gate) * up (each times the pair's input
// weight first, if there is one); 2: out = relu(product)^2.
template <int MODE>
__global__ void __launch_bounds__(MT_THREADS, 1)
moe_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x16,
                   const __grid_constant__ CUtensorMap map_x64, const __grid_constant__ CUtensorMap map_x128, const __grid_constant__ CUtensorMap map_out, MoeTcArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* staging = smem + MT_STAGES * MT_STAGE_BYTES;
    uint64_t* bars = (uint64_t*)(staging + 2 * MT_OUT_BYTES);
    uint64_t* full = bars;                                  // counted in the leader only
    uint64_t* empty = bars + MT_STAGES;                     // one in each CTA, for its own loader
    uint64_t* acc_full = bars + 2 * MT_STAGES;              // [2], one in each CTA, for its own epilogue
    uint64_t* acc_empty = acc_full + 2;                     // [2], counted in the leader: both CTAs' epilogues
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const bool leader = rank == 0;
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x16) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x64) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x128) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_out) : "memory");
        for (int s = 0; s < MT_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * 128); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(tmem_slot, MT_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                       // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();                               // the plan says which weights this CTA reads

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            MtWalk walk(a);
            MtUnit t;
            int issued = 0;
            while (ok && walk.next(t)) {
                const int half = t.chunks * (MT_CHUNK / 2);              // slots of this CTA's half
                const int box = half <= 16 ? 16 : half <= 64 ? 64 : 128;  // a box may reach into the next slots: nothing reads those
                const CUtensorMap* map_x = box == 16 ? &map_x16 : box == 64 ? &map_x64 : &map_x128;
                const uint32_t bytes = 2 * (MT_A_BYTES + box * MT_BLOCK_K * 2);
                const int wy = t.expert * a.w_rows + t.m0 + (int)rank * MT_BLOCK_M, xy = t.slot0 + (int)rank * half;
                for (int i = 0; i < a.total_kb; ++i, ++issued) {
                    uint8_t* sa = smem + stage * MT_STAGE_BYTES;
                    if (issued >= MT_STAGES) {
                        ok = mbar_wait(&empty[stage], phase ^ 1u, abort_flag);
                        if (!ok) break;
                    }
                    if (leader) mbar_expect_tx(&full[stage], bytes);
                    tma_load_2d_pair(&map_w, &full[stage], sa, i * MT_BLOCK_K, wy);
                    tma_load_2d_pair(map_x, &full[stage], sa + MT_A_BYTES, i * MT_BLOCK_K, xy);
                    if (++stage == MT_STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            int stage = 0, buf = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            MtWalk walk(a);
            MtUnit t;
            while (ok && walk.next(t)) {
                const uint32_t idesc = umma_idesc_bf16(2 * MT_BLOCK_M, t.chunks * MT_CHUNK);
                ok = mbar_wait(&acc_empty[buf], ((acc_phase >> buf) & 1u) ^ 1u, abort_flag);   // both epilogues have drained it
                if (!ok) break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + buf * 256;
                for (int i = 0; i < a.total_kb; ++i) {
                    ok = mbar_wait(&full[stage], phase, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + stage * MT_STAGE_BYTES);
                    const uint32_t sb = sa + MT_A_BYTES;
#pragma unroll
                    for (int k = 0; k < MT_BLOCK_K / MT_UMMA_K; ++k) {
                        const uint32_t koff = k * MT_UMMA_K * 2;
                        umma_bf16_pair(tmem_d, umma_desc_sw128(sa + koff), umma_desc_sw128(sb + koff), idesc, (i > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit_pair(&empty[stage]);
                    if (++stage == MT_STAGES) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                umma_commit_pair(&acc_full[buf]);
                acc_phase ^= (1u << buf);
                buf ^= 1;
            }
        }
    } else {
        const int quarter = warp & 3;
        const bool issuer = threadIdx.x == 64;             // the one thread that issues and awaits the TMA stores
        int buf = 0;
        uint32_t full_phase = 0, chunk_no = 0;
        bool ok = true;
        MtWalk walk(a);
        MtUnit t;
        while (ok && walk.next(t)) {
            const int m0 = t.m0 + (int)rank * MT_BLOCK_M;                  // this CTA's 128 rows of the pair's 256
            ok = epilogue_all(mbar_wait(&acc_full[buf], (full_phase >> buf) & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
            const uint32_t trow = tmem_base + buf * 256 + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < t.chunks; ++c) {
                float v[MT_CHUNK];
                tmem_ld32(trow + c * MT_CHUNK, v);
                // the staging tile is free once the store before the last one has read it
                uint8_t* tile = staging + (chunk_no & 1u) * MT_OUT_BYTES;
                ++chunk_no;
                if (issuer) bulk_wait_read_1();
                epilogue_sync();
                if (MODE == 1) {
                    // [32 slots][64 outputs]; the halves of a warp hold gate and up rows and swap values
                    float wi = 1.f;
                    if (a.in_wgt) {
                        const int pair = a.slot_pair[t.slot0 + c * MT_CHUNK + lane];
                        wi = pair >= 0 ? a.in_wgt[pair] : 0.f;
                    }
                    const bool is_up = (lane & 16) != 0;
                    __nv_bfloat16* dst = (__nv_bfloat16*)tile + (is_up ? 64 : 0) + quarter * 16 + (lane & 15);
#pragma unroll
                    for (int p2 = 0; p2 < MT_CHUNK / 2; ++p2) {
                        const float from_up = __shfl_xor_sync(0xffffffffu, v[2 * p2], 16);
                        const float from_gate = __shfl_xor_sync(0xffffffffu, v[2 * p2 + 1], 16);
                        const float w2 = __shfl_sync(0xffffffffu, wi, 2 * p2 + (is_up ? 1 : 0));
                        const float g = (is_up ? from_gate : v[2 * p2]) * w2;
                        const float u = (is_up ? v[2 * p2 + 1] : from_up) * w2;
                        dst[2 * p2 * 64] = __float2bfloat16_rn(silu_to_bf16(g) * u);
                    }
                } else {
                    __nv_bfloat16* dst = (__nv_bfloat16*)tile + quarter * 32 + lane;
#pragma unroll
                    for (int i = 0; i < MT_CHUNK; ++i) {
                        const float r = MODE == 2 ? fmaxf(v[i], 0.f) : v[i];
                        dst[i * MT_BLOCK_M] = __float2bfloat16_rn(MODE == 2 ? r * r : r);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                epilogue_sync();
                const int x0 = MODE == 1 ? m0 / 2 : m0;
                if (issuer && x0 < a.m_out) {              // columns past the matrix are clipped by the tensor map
                    tma_store_2d(&map_out, tile, x0, t.slot0 + c * MT_CHUNK);
                    bulk_commit();
                }
            }
            tc_fence_before();
            mbar_arrive_leader(&acc_empty[buf]);
            full_phase ^= (1u << buf);
            buf ^= 1;
        }
        if (issuer) bulk_wait_all();                       // the stores are complete, not only read, before the kernel ends
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicExch(a.error_flag, 1);
    cluster_sync_all();                       // neither CTA frees tensor memory or leaves while the other may still signal it
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, MT_TMEM_COLS);
    }
}

// The slots' rows: xs[slot] = x[token of the slot], zeros for padding slots.  A warp a slot, 16 bytes a lane.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* __restrict__ x, uint4* __restrict__ xs, const int* __restrict__ slot_pair, const int* __restrict__ meta,
                  long long ldx16, int k16, int top) {
    pdl_trigger();
    pdl_wait();
    const int slot = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (slot >= meta[0] * MT_CHUNK) return;
    const int pair = slot_pair[slot];
    const uint4* src = x + (size_t)(pair >= 0 ? pair / top : 0) * ldx16;
    uint4* dst = xs + (size_t)slot * k16;
#pragma unroll 8
    for (int i = threadIdx.x & 31; i < k16; i += 32) dst[i] = pair >= 0 ? src[i] : make_uint4(0, 0, 0, 0);
}

// Slots of MT_CHUNK * max_tiles; rows of k elements.
extern "C" int braid_moe_gather(const void* x, void* xs, const int* slot_pair, const int* meta, long long ldx, int k, int top,
                                int max_tiles, void* stream) {
    if (max_tiles <= 0) return BRAID_OK;
    if (k <= 0 || k % 8 || ldx % 8 || (((uintptr_t)x | (uintptr_t)xs) & 15)) BRAID_REFUSE("moe_gather: rows of %d elements, %lld apart, must be whole runs of 16 bytes", k, ldx);
    braid_launch(moe_gather_kernel, dim3(max_tiles * (MT_CHUNK / 8)), dim3(256), 0, (cudaStream_t)stream, (const uint4*)x, (uint4*)xs,
                 slot_pair, meta, ldx / 8, k / 8, top);
    BRAID_LAUNCH_CHECK();
}

static int mt_map(CUtensorMap* map, const void* base, long long inner, long long rows, long long ld, int box_inner, int box_rows, bool swizzle) {
    TcEncodeTiledFn fn = tc_encode_tiled_fn();
    if (!fn) BRAID_REFUSE("moe_gemm_tc: the driver does not export cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                    swizzle ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) BRAID_REFUSE("moe_gemm_tc: cuTensorMapEncodeTiled failed with %d (inner=%lld rows=%lld ld=%lld)", (int)r, inner, rows, ld);
    return BRAID_OK;
}

template <int MODE>
static int launch_moe_tc(const CUtensorMap& mw, const CUtensorMap& x16, const CUtensorMap& x64, const CUtensorMap& x128, const CUtensorMap& mo, const MoeTcArgs& a,
                         int pairs, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(moe_gemm_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM_BYTES);
        if (e != cudaSuccess) { braid_set_error("moe_gemm_tc: cannot reserve %d bytes of shared memory: %s", MT_SMEM_BYTES, cudaGetErrorString(e)); return (int)e; }
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(MT_THREADS);
    cfg.dynamicSmemBytes = MT_SMEM_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = braid_pdl_enabled();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, moe_gemm_tc_kernel<MODE>, mw, x16, x64, x128, mo, a);
    BRAID_LAUNCH_CHECK();
}

// x [max_tiles * 32 slots, k]; w: experts x w_rows rows of k (mode 1: gate and up interleaved in blocks of 16 rows, w_rows =
// 2 * (m_out rounded up to 16); else w_rows = m_out); out [slots, ldo], its first m_out columns.
extern "C" int braid_moe_gemm_tc(const void* x, const void* w, void* out, const int* slot_pair, const int* tile_expert, const int* wide,
                                 const int* meta, int mode, int experts, int w_rows, int m_out, int k, long long ldo, int max_tiles,
                                 int max_wide, const float* in_wgt, int* error_flag, void* stream) {
    if (max_tiles <= 0 || m_out <= 0) return BRAID_OK;
    if (mode < 0 || mode > 2) BRAID_REFUSE("moe_gemm_tc: unknown mode %d", mode);
    if (k <= 0 || k % 8 || ldo % 8 || ldo < m_out) BRAID_REFUSE("moe_gemm_tc: k=%d and the output's stride %lld must be multiples of 8", k, ldo);
    if ((((uintptr_t)x | (uintptr_t)w | (uintptr_t)out | (uintptr_t)wide) & 15)) BRAID_REFUSE("moe_gemm_tc: operands must start on 16 bytes");
    if (w_rows != (mode == 1 ? 2 * ((m_out + 15) / 16 * 16) : m_out)) BRAID_REFUSE("moe_gemm_tc: %d weight rows an expert do not fit %d outputs", w_rows, m_out);
    if (in_wgt && mode != 1) BRAID_REFUSE("moe_gemm_tc: a weight on the expert's input goes with the gated first product");
    if (!error_flag) BRAID_REFUSE("moe_gemm_tc: error_flag is required");
    const long long slots = (long long)max_tiles * MT_CHUNK;
    CUtensorMap mw, x16, x64, x128, mo;
    int rc = mt_map(&mw, w, k, (long long)experts * w_rows, k, MT_BLOCK_K, 128, true);
    if (!rc) rc = mt_map(&x16, x, k, slots, k, MT_BLOCK_K, 16, true);
    if (!rc) rc = mt_map(&x64, x, k, slots, k, MT_BLOCK_K, 64, true);
    if (!rc) rc = mt_map(&x128, x, k, slots, k, MT_BLOCK_K, 128, true);
    if (!rc) rc = mt_map(&mo, out, m_out, slots, ldo, mode == 1 ? MT_BLOCK_M / 2 : MT_BLOCK_M, MT_CHUNK, false);
    if (rc) return rc;
    const int m_tiles = (w_rows + 2 * MT_BLOCK_M - 1) / (2 * MT_BLOCK_M);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 1) sms = 148;
    const long long units = (long long)m_tiles * max_wide;
    const int pairs = (int)(units < sms / 2 ? units : sms / 2);
    MoeTcArgs a{tile_expert, (const int4*)wide, meta, slot_pair, in_wgt, m_tiles, w_rows, (k + MT_BLOCK_K - 1) / MT_BLOCK_K, m_out, max_wide, error_flag};
    cudaStream_t s = (cudaStream_t)stream;
    if (mode == 0) return launch_moe_tc<0>(mw, x16, x64, x128, mo, a, pairs, s);
    if (mode == 1) return launch_moe_tc<1>(mw, x16, x64, x128, mo, a, pairs, s);
    return launch_moe_tc<2>(mw, x16, x64, x128, mo, a, pairs, s);
}
