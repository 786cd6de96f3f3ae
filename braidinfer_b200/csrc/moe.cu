// Mixture of experts: routing, the plan that sorts a step's (token, choice) pairs by expert, the
// experts' matrix products over those sorted rows, and the weighted sum back into the residual stream.
//
// Routing (one warp a token): s = softmax(z) over all experts; the experts form `groups` equal groups of
// neighbours, a group's score is its largest s, and only experts of the `keep` best groups can be chosen;
// the `top` allowed experts with the largest s are chosen (ties: the lower index); their weights are
// their s divided by the sum of the chosen s (+ 1e-20), times `mult` (a constant factor the caller wants
// on the layer's output).  Everything float32.  `sigmoid` routing instead scores every expert by itself,
// s = 1 / (1 + exp(-z)), chooses the same way, and leaves the chosen scores as the weights (times `mult`), not
// renormalised.  With `correction` (a number an expert) the choice is made on score + correction while the weights keep
// the scores without it; `renorm` says whether the weights are divided by their sum.
//
// The plan: every chosen (token, choice) pair gets a slot in an array ordered by expert, each expert's run
// padded to a multiple of `tile` slots, so that a tile of slots belongs to one expert and the products can
// run tile by tile with the sizes known only on the device.  Which slot of its expert's run a pair gets
// does not touch any number: every output row is a sum over k in a fixed order whatever its slot.
// Launch sizes depend on the step's shape alone (an upper bound of tiles), so a CUDA graph can replay them.
#include "common.cuh"
#include "mma_tile.cuh"

// ------------------------------------------------------------------ routing
struct MoeRouteArgs {
    const float* logits;      // [rows, experts]
    int* idx;                 // [rows, top]
    float* wgt;               // [rows, top]
    int rows, experts, top, groups, keep;
    float mult;
    int sigmoid;              // scores are sigmoids of the logits, not their softmax
    int renorm;               // the chosen scores are divided by their sum
    const float* correction;  // [experts] float32, added to the scores for the choice alone; or null
};

#define MOE_ROUTE_WARPS 4

__global__ void __launch_bounds__(MOE_ROUTE_WARPS * 32)
moe_route_kernel(MoeRouteArgs a) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float smem[];          // per warp: [experts] scores, [groups] group scores, [experts] choice scores
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * MOE_ROUTE_WARPS + warp;
    if (row >= a.rows) return;
    float* s = smem + (size_t)warp * (2 * a.experts + a.groups);
    float* gs = s + a.experts;
    float* cs = gs + a.groups;               // what the choice is made on: -inf once an expert is chosen
    const float* z = a.logits + (size_t)row * a.experts;
    if (a.sigmoid) {
        for (int e = lane; e < a.experts; e += 32) s[e] = 1.f / (1.f + expf(-z[e]));
    } else {
        float mx = -INFINITY;
        for (int e = lane; e < a.experts; e += 32) mx = fmaxf(mx, z[e]);
        mx = warp_max(mx);
        float sum = 0.f;
        for (int e = lane; e < a.experts; e += 32) {
            const float p = expf(z[e] - mx);
            s[e] = p;
            sum += p;
        }
        sum = warp_sum(sum);
        const float inv = 1.f / sum;
        for (int e = lane; e < a.experts; e += 32) s[e] *= inv;
    }
    for (int e = lane; e < a.experts; e += 32) cs[e] = a.correction ? s[e] + a.correction[e] : s[e];   // this lane's own scores
    __syncwarp();
    const int per = a.experts / a.groups;
    for (int g = lane; g < a.groups; g += 32) {
        float m = -INFINITY;
        for (int i = 0; i < per; ++i) m = fmaxf(m, s[g * per + i]);
        gs[g] = m;
    }
    __syncwarp();
    // the `keep` best groups stay; the others are closed by marking their score negative
    // (a kept group's score is made > 2, a softmax score never is)
    for (int k = 0; k < a.keep; ++k) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int g = lane; g < a.groups; g += 32) {
            const float v = gs[g];
            if (v <= 2.f && (v > best || (v == best && g < bi))) { best = v; bi = g; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0 && bi != 0x7fffffff) gs[bi] = 3.f;
        __syncwarp();
    }
    // the `top` largest scores among experts of kept groups; a chosen expert's choice score is then hidden
    float chosen_sum = 0.f;
    for (int k = 0; k < a.top; ++k) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < a.experts; e += 32) {
            const float v = cs[e];
            if (v > -INFINITY && gs[e / per] > 2.f && (v > best || (v == best && e < bi))) { best = v; bi = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (bi == 0x7fffffff) bi = -1;                      // fewer allowed experts than `top`
        best = bi >= 0 ? s[bi] : 0.f;                       // the weight is the score without the correction
        if (lane == 0) {
            a.idx[(size_t)row * a.top + k] = bi;
            a.wgt[(size_t)row * a.top + k] = best;
            if (bi >= 0) cs[bi] = -INFINITY;
        }
        chosen_sum += best;
        __syncwarp();
    }
    const float norm = a.renorm ? a.mult / (chosen_sum + 1e-20f) : a.mult;
    __syncwarp();
    for (int k = lane; k < a.top; k += 32) a.wgt[(size_t)row * a.top + k] *= norm;
}

extern "C" int braid_moe_route(const float* logits, int* idx, float* wgt, int rows, int experts, int top,
                               int groups, int keep, float mult, int sigmoid, int renorm, const float* correction,
                               void* stream) {
    if (rows <= 0) return BRAID_OK;
    if (experts <= 0 || top <= 0 || top > experts) BRAID_REFUSE("moe_route: top=%d of %d experts", top, experts);
    if (groups <= 0 || experts % groups || keep <= 0 || keep > groups) BRAID_REFUSE("moe_route: %d experts in %d groups, %d kept", experts, groups, keep);
    if (correction && groups != 1) BRAID_REFUSE("moe_route: a correction of the choice is built for experts in one group, not %d", groups);
    const size_t smem = (size_t)MOE_ROUTE_WARPS * (2 * experts + groups) * sizeof(float);
    if (smem > 48 * 1024) BRAID_REFUSE("moe_route: %d experts are more than one block's shared memory holds", experts);
    MoeRouteArgs a{logits, idx, wgt, rows, experts, top, groups, keep, mult, sigmoid, renorm, correction};
    braid_launch(moe_route_kernel, dim3((rows + MOE_ROUTE_WARPS - 1) / MOE_ROUTE_WARPS), dim3(MOE_ROUTE_WARPS * 32), smem,
                 (cudaStream_t)stream, a);
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ the plan
// One cluster.  idx [rows * top] holds each pair's expert (-1: none); pairs of padding rows (token_seq < 0)
// take no slot.  Outputs: slot_pair [cap] (pair of each slot, -1 for padding slots), pair_slot [rows * top]
// (slot of each pair, -1 for none), tile_expert [max_tiles], meta[0] = tiles in use.  With `wide` (tiles of 32 slots, moe_tc.cu):
// an expert's tiles in runs of up to eight, shared out evenly: {first slot, tiles, the expert's first run, its runs} a run,
// meta[1] = runs in use.
// Bound by latency: two passes over the pairs (four loads in flight a thread, a shared-memory atomic a pair), shared by the CTAs of
// one cluster, which read each other's counts, and two sums over the experts by shuffles.
#define MOE_MAX_EXPERTS 1024
#define MOE_PLAN_BATCH 4
#define MOE_WIDE_TILES 8

// the sums of a and b over the threads before this one; *total_* over all of them (1,024 threads)
__device__ __forceinline__ void moe_scan2(int& a, int& b, int* total_a, int* total_b, int* warp_a, int* warp_b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ta = __shfl_up_sync(0xffffffffu, ia, o), tb = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) { ia += ta; ib += tb; }
    }
    if (lane == 31) { warp_a[warp] = ia; warp_b[warp] = ib; }
    __syncthreads();
    int wa = warp_a[lane], wb = warp_b[lane];
    const int own_a = wa, own_b = wb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ta = __shfl_up_sync(0xffffffffu, wa, o), tb = __shfl_up_sync(0xffffffffu, wb, o);
        if (lane >= o) { wa += ta; wb += tb; }
    }
    *total_a = __shfl_sync(0xffffffffu, wa, 31);
    *total_b = __shfl_sync(0xffffffffu, wb, 31);
    a = ia - a + __shfl_sync(0xffffffffu, wa - own_a, warp);
    b = ib - b + __shfl_sync(0xffffffffu, wb - own_b, warp);
}
// the last e with start[e] <= t among those that own anything (start is not falling; start[experts] is the total)
__device__ __forceinline__ int moe_owner(const int* start, int experts, int t) {
    int lo = 0, hi = experts;                               // start[lo] <= t < start[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}
// the number at `p` (this CTA's shared memory) in CTA `rank` of the cluster
__device__ __forceinline__ int moe_peer_load(const int* p, int rank) {
    uint32_t at;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void moe_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(1024)
moe_plan_kernel(const int* __restrict__ idx, const int* __restrict__ token_seq, int* __restrict__ slot_pair,
                int* __restrict__ pair_slot, int* __restrict__ tile_expert, int* __restrict__ meta, int4* __restrict__ wide,
                int rows, int top, int experts, int tile, int max_tiles, int max_wide) {
    pdl_trigger();
    pdl_wait();
    __shared__ int count[MOE_MAX_EXPERTS], cursor[MOE_MAX_EXPERTS], start[MOE_MAX_EXPERTS + 1], start_w[MOE_MAX_EXPERTS + 1],
        warp_a[32], warp_b[32];
    const int pairs = rows * top, tid = threadIdx.x, ctas = gridDim.x, rank = blockIdx.x;      // the grid is one cluster
    const int all = ctas * 1024, at = rank * 1024 + tid;
    count[tid] = 0;
    for (int i = at; i < max_tiles * tile; i += all) slot_pair[i] = -1;
    __syncthreads();
    auto fetch = [&](int base, int* e) {
#pragma unroll
        for (int j = 0; j < MOE_PLAN_BATCH; ++j) {
            const int i = base + j * all + at;
            e[j] = -1;
            if (i < pairs) {
                const int want = idx[i], seq = token_seq[i / top];
                if (seq >= 0 && want >= 0 && want < experts) e[j] = want;
            }
        }
    };
    for (int base = 0; base < pairs; base += MOE_PLAN_BATCH * all) {
        int e[MOE_PLAN_BATCH];
        fetch(base, e);
#pragma unroll
        for (int j = 0; j < MOE_PLAN_BATCH; ++j)
            if (e[j] >= 0) atomicAdd(&count[e[j]], 1);
    }
    if (ctas > 1) moe_cluster_sync(); else __syncthreads();
    // an expert's pairs over all CTAs, and those of the CTAs before this one
    int total = 0, before = 0;
    if (tid < experts) {
        if (ctas == 1) total = count[tid];
        else
            for (int r = 0; r < ctas; ++r) {
                const int n = moe_peer_load(&count[tid], r);
                if (r < rank) before += n;
                total += n;
            }
    }
    cursor[tid] = before;
    int tiles, wides, s = (total + tile - 1) / tile, w = (s + MOE_WIDE_TILES - 1) / MOE_WIDE_TILES;
    moe_scan2(s, w, &tiles, &wides, warp_a, warp_b);
    start[tid] = s;
    start_w[tid] = w;
    if (tid == 0) {
        start[MOE_MAX_EXPERTS] = tiles;
        start_w[MOE_MAX_EXPERTS] = wides;
        if (rank == 0) {
            meta[0] = tiles < max_tiles ? tiles : max_tiles;
            if (wide) meta[1] = wides < max_wide ? wides : max_wide;
        }
    }
    if (ctas > 1) moe_cluster_sync(); else __syncthreads();              // nobody leaves while its counts are read
    for (int t = at; t < tiles && t < max_tiles; t += all) tile_expert[t] = moe_owner(start, experts, t);
    if (wide)
        for (int t = at; t < wides && t < max_wide; t += all) {
            const int e = moe_owner(start_w, experts, t), first = start_w[e], runs = start_w[e + 1] - first, n = start[e + 1] - start[e];
            const int lo = (t - first) * n / runs, hi = (t - first + 1) * n / runs;
            wide[t] = make_int4((start[e] + lo) * tile, hi - lo, first, runs);
        }
    for (int base = 0; base < pairs; base += MOE_PLAN_BATCH * all) {
        int e[MOE_PLAN_BATCH];
        fetch(base, e);
#pragma unroll
        for (int j = 0; j < MOE_PLAN_BATCH; ++j) {
            const int i = base + j * all + at;
            if (i >= pairs) break;
            int slot = e[j] >= 0 ? start[e[j]] * tile + atomicAdd(&cursor[e[j]], 1) : -1;
            if (slot >= max_tiles * tile) slot = -1;
            if (slot >= 0) slot_pair[slot] = i;
            pair_slot[i] = slot;
        }
    }
}

extern "C" int braid_moe_plan(const int* idx, const int* token_seq, int* slot_pair, int* pair_slot, int* tile_expert,
                              int* meta, int* wide, int rows, int top, int experts, int tile, int max_tiles, int max_wide, void* stream) {
    if (rows <= 0) return BRAID_OK;
    if (experts <= 0 || experts > MOE_MAX_EXPERTS) BRAID_REFUSE("moe_plan: %d experts (at most %d)", experts, MOE_MAX_EXPERTS);
    if (tile <= 0 || tile % 16) BRAID_REFUSE("moe_plan: the tile of %d slots must be a multiple of 16", tile);
    if (wide && ((uintptr_t)wide & 15)) BRAID_REFUSE("moe_plan: the runs of tiles must start on 16 bytes");
    // one CTA for a decode step's pairs, up to a cluster of eight
    const long long pairs = (long long)rows * top;
    const int ctas = pairs <= 1024 ? 1 : pairs <= 2048 ? 2 : pairs <= 4096 ? 4 : 8;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(1024);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = braid_pdl_enabled();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, moe_plan_kernel, idx, token_seq, slot_pair, pair_slot, tile_expert, meta, (int4*)wide, rows, top, experts,
                       tile, max_tiles, max_wide);
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ routing and plan of a few tokens
// moe_route_kernel and moe_plan_kernel of a step of up to 8 tokens in one CTA: a warp routes a token, and with no expert above 8 pairs a
// plan is bits: an expert's tile is the number of chosen experts below it, a pair's slot in it the number of earlier tokens that chose it.
// Bound by latency (some hundred numbers): a lane holds its experts' scores in registers, and a choice is two warp-wide reductions, the
// largest score's bits, then the lowest of the experts that have them, instead of ten shuffles.  The same numbers as the two kernels:
// the sums are taken in their order.  8 tokens, 6 of 64 experts in 8 groups: 7.2 us and 3.8 in a step's chain, this 3.9
// (4 tokens, 64 experts in one group: 4.1 and 3.5, this 3.2).  Larger steps keep the two kernels, whose CTAs share the tokens.
#define MOE_RP_TOKENS 8
#define MOE_RP_EXPERTS 256
#define MOE_RP_TILE 32

// A number's place among the floats, as an integer above 0; 0 for what can't be chosen (-inf, NaN).
__device__ __forceinline__ uint32_t moe_key(float v) {
    const uint32_t b = __float_as_uint(v + 0.f);             // (-0 and 0 are one)
    return !(v > -INFINITY) ? 0u : (b & 0x80000000u) ? ~b : b | 0x80000000u;
}

template <int R>
__global__ void __launch_bounds__(MOE_RP_TOKENS * 32)
moe_route_plan_kernel(MoeRouteArgs a, const int* __restrict__ token_seq, int* __restrict__ slot_pair, int* __restrict__ pair_slot,
                      int* __restrict__ tile_expert, int* __restrict__ meta, int4* __restrict__ wide, int max_tiles, int max_wide) {
    pdl_trigger();
    __shared__ uint32_t chosen[MOE_RP_EXPERTS / 32];         // a bit an expert
    __shared__ uint32_t who[MOE_RP_EXPERTS];                 // an expert's tokens, a bit each
    __shared__ float group_s[MOE_RP_TOKENS][MOE_RP_EXPERTS];
    const int tid = threadIdx.x, row = tid >> 5, lane = tid & 31;
    const bool live = row < a.rows;
    who[tid] = 0;
    if (tid < MOE_RP_EXPERTS / 32) chosen[tid] = 0;
    const bool placed = live && token_seq[row] >= 0;         // the step's tables are there before its first kernel
    pdl_wait();
    for (int i = tid; i < max_tiles * MOE_RP_TILE; i += MOE_RP_TOKENS * 32) slot_pair[i] = -1;
    __syncthreads();
    int mine = -1;                                           // lane k: choice k
    if (live) {
        const float* z = a.logits + (size_t)row * a.experts;
        float s[R];
        uint32_t key[R];
#pragma unroll
        for (int i = 0; i < R; ++i) s[i] = lane + 32 * i < a.experts ? z[lane + 32 * i] : -INFINITY;
        if (a.sigmoid) {
#pragma unroll
            for (int i = 0; i < R; ++i) s[i] = 1.f / (1.f + expf(-s[i]));
        } else {
            float mx = -INFINITY, sum = 0.f;
#pragma unroll
            for (int i = 0; i < R; ++i) mx = fmaxf(mx, s[i]);
            mx = warp_max(mx);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (lane + 32 * i < a.experts) { s[i] = expf(s[i] - mx); sum += s[i]; }
            const float inv = 1.f / warp_sum(sum);
#pragma unroll
            for (int i = 0; i < R; ++i) s[i] *= inv;
        }
        uint32_t kept = 0xffffffffu;                         // a bit a group
        const int per = a.experts / a.groups;
        if (a.keep < a.groups) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (lane + 32 * i < a.experts) group_s[row][lane + 32 * i] = s[i];
            __syncwarp();
            float m = -INFINITY;
            if (lane < a.groups)
                for (int i = 0; i < per; ++i) m = fmaxf(m, group_s[row][lane * per + i]);
            // one above an expert's key: a group whose scores are no numbers is still a group
            uint32_t gk = lane < a.groups ? moe_key(m) + 1u : 0u;
            for (int k = 0; k < a.keep; ++k) {
                const uint32_t best = __reduce_max_sync(0xffffffffu, gk);
                const uint32_t who_best = __ballot_sync(0xffffffffu, gk == best);
                if (lane == __ffs(who_best) - 1) gk = 0u;
            }
            kept = __ballot_sync(0xffffffffu, lane < a.groups && gk == 0u);
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int e = lane + 32 * i;
            key[i] = 0u;
            if (e < a.experts && (a.keep >= a.groups || (kept >> (e / per)) & 1u)) key[i] = moe_key(a.correction ? s[i] + a.correction[e] : s[i]);
        }
        float chosen_sum = 0.f, my_w = 0.f;
        for (int k = 0; k < a.top; ++k) {
            uint32_t bk = 0u;
            int be = 0;
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (key[i] > bk) { bk = key[i]; be = i; }    // an equal one further up waits
            const uint32_t best = __reduce_max_sync(0xffffffffu, bk);
            const int e = best ? (int)__reduce_min_sync(0xffffffffu, bk == best ? (uint32_t)(lane + 32 * be) : 0xffffffffu) : -1;
            float w = 0.f;
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (e == lane + 32 * i) { w = s[i]; key[i] = 0u; }
            w = e >= 0 ? __shfl_sync(0xffffffffu, w, e & 31) : 0.f;
            if (lane == k) { mine = e; my_w = w; }
            chosen_sum += w;
        }
        const float norm = a.renorm ? a.mult / (chosen_sum + 1e-20f) : a.mult;
        if (lane < a.top) {
            a.idx[(size_t)row * a.top + lane] = mine;
            a.wgt[(size_t)row * a.top + lane] = my_w * norm;
        }
        if (!placed) mine = -1;
        if (mine >= 0) {
            atomicOr(&who[mine], 1u << row);
            atomicOr(&chosen[mine >> 5], 1u << (mine & 31));
        }
    }
    __syncthreads();
    auto below = [&](int e) {                                // chosen experts before e
        int n = __popc(chosen[e >> 5] & ((1u << (e & 31)) - 1u));
        for (int i = 0; i < (e >> 5); ++i) n += __popc(chosen[i]);
        return n;
    };
    if (live && lane < a.top) {
        const int pair = row * a.top + lane;
        int slot = mine >= 0 ? below(mine) * MOE_RP_TILE + __popc(who[mine] & ((1u << row) - 1u)) : -1;
        if (slot >= max_tiles * MOE_RP_TILE) slot = -1;
        if (slot >= 0) slot_pair[slot] = pair;
        pair_slot[pair] = slot;
    }
    if (who[tid]) {
        const int t = below(tid);
        if (t < max_tiles) tile_expert[t] = tid;
        if (t < max_wide) wide[t] = make_int4(t * MOE_RP_TILE, 1, t, 1);
    }
    if (tid == 0) {
        int n = 0;
        for (int i = 0; i < MOE_RP_EXPERTS / 32; ++i) n += __popc(chosen[i]);
        meta[0] = n < max_tiles ? n : max_tiles;
        meta[1] = n < max_wide ? n : max_wide;
    }
}

extern "C" int braid_moe_route_plan(const float* logits, int* idx, float* wgt, int rows, int experts, int top, int groups, int keep, float mult,
                                    int sigmoid, int renorm, const float* correction, const int* token_seq, int* slot_pair, int* pair_slot,
                                    int* tile_expert, int* meta, int* wide, int max_tiles, int max_wide, void* stream) {
    if (rows <= 0) return BRAID_OK;
    if (experts <= 0 || top <= 0 || top > experts) BRAID_REFUSE("moe_route_plan: top=%d of %d experts", top, experts);
    if (groups <= 0 || experts % groups || keep <= 0 || keep > groups) BRAID_REFUSE("moe_route_plan: %d experts in %d groups, %d kept", experts, groups, keep);
    if (correction && groups != 1) BRAID_REFUSE("moe_route_plan: a correction of the choice is built for experts in one group, not %d", groups);
    if (rows > MOE_RP_TOKENS || experts > MOE_RP_EXPERTS || top > 32 || groups > 32)
        BRAID_REFUSE("moe_route_plan: %d rows, %d choices of %d experts in %d groups are more than one CTA takes", rows, top, experts, groups);
    if (!wide || ((uintptr_t)wide & 15)) BRAID_REFUSE("moe_route_plan: the runs of tiles must start on 16 bytes");
    const MoeRouteArgs a{logits, idx, wgt, rows, experts, top, groups, keep, mult, sigmoid, renorm, correction};
    cudaStream_t s = (cudaStream_t)stream;
#define ROUTE_PLAN(R) braid_launch(moe_route_plan_kernel<R>, dim3(1), dim3(MOE_RP_TOKENS * 32), 0, s, a, token_seq, slot_pair, pair_slot, \
                                   tile_expert, meta, (int4*)wide, max_tiles, max_wide)
    if (experts <= 64) ROUTE_PLAN(2);
    else ROUTE_PLAN(8);
#undef ROUTE_PLAN
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ the experts' products, plain
// Units of 16 slots x 64 outputs; 256 threads, each one slot and four outputs; float32 FMA in a fixed
// order along k.  MODE 0: act[slot, j] = silu(x[token] . gate_e[j]) * (x[token] . up_e[j]), the input rows
// gathered through slot_pair.  MODE 1: y[slot, j] = act[slot] . down_e[j].  MODE 2 (experts without a gate):
// act[slot, j] = relu(x[token] . up_e[j])^2, the input rows gathered like MODE 0's, w0 the up matrices.
// With `in_wgt` (MODE 0) a pair's weight multiplies the expert's input instead of its output: the expert sees w x, and
// since its first products are linear, gate and up are multiplied by w in float32 before the activation,
// act = silu(w (x . gate)) * (w (x . up)); the weighted sum then adds the pairs with weight 1.
struct MoeGemmArgs {
    const void* x;            // MODE 0: [rows, ldx] the layer's normed input; MODE 1: act [slots, ldx]
    const void* w0;           // MODE 0: gate [experts, J, K]; MODE 1: down [experts, J, K]
    const void* w1;           // MODE 0: up [experts, J, K]
    void* out;                // [slots, ldo]
    const int* slot_pair;
    const int* tile_expert;
    const int* meta;
    long long ldx, ldo;
    int J, K, top, tile;
    const float* in_wgt;      // MODE 0: [rows * top] a weight a pair on the expert's input; or null
    long long we, wb;         // elements from an expert's rows to the next one's, and from 16 of its rows to the next 16
};

// Row m of expert e: rows lie K apart in blocks of 16, the blocks `wb` apart (16 K where nothing lies between them).
template <typename T>
__device__ __forceinline__ const T* moe_weight_row(const MoeGemmArgs& a, const void* w, int e, int m) {
    return (const T*)w + (size_t)e * a.we + (size_t)(m >> 4) * a.wb + (size_t)(m & 15) * a.K;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(256)
moe_gemm_simt_kernel(MoeGemmArgs a) {
    pdl_trigger();
    pdl_wait();
    __shared__ float xs[16][16 + 1];        // [k][slot]
    __shared__ float w0s[16][64 + 4];       // [k][output]
    __shared__ float w1s[MODE == 0 ? 16 : 1][64 + 4];
    const int unit = blockIdx.y;                             // 16 slots
    const int t = unit * 16 / a.tile;
    if (t >= a.meta[0]) return;
    const int e = a.tile_expert[t];
    const int slot0 = unit * 16;
    const int m0 = blockIdx.x * 64;
    const int ts = threadIdx.x >> 4, tj = threadIdx.x & 15;  // ts: slot, tj: group of four outputs
    const int my_pair = a.slot_pair[slot0 + ts];
    // the row this thread fetches for the x tile: thread (r = tid >> 4, c = tid & 15) loads x[slot r][k0 + c]
    const long long src_row = (MODE != 1) ? (my_pair >= 0 ? my_pair / a.top : -1) : (slot0 + ts);
    float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0; k0 < a.K; k0 += 16) {
        {
            const int k = k0 + tj;
            xs[tj][ts] = (src_row >= 0 && k < a.K) ? to_f32(((const T*)a.x)[(size_t)src_row * a.ldx + k]) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int el = threadIdx.x + i * 256;            // 0..1023: 64 outputs x 16 k
            const int r = el >> 4, c = el & 15;
            const int k = k0 + c, m = m0 + r;
            const bool ok = (m < a.J && k < a.K);
            w0s[c][r] = ok ? to_f32(moe_weight_row<T>(a, a.w0, e, m)[k]) : 0.f;
            if (MODE == 0) w1s[c][r] = ok ? to_f32(moe_weight_row<T>(a, a.w1, e, m)[k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const float xv = xs[kk][ts];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc0[j] = fmaf(xv, w0s[kk][tj * 4 + j], acc0[j]);
                if (MODE == 0) acc1[j] = fmaf(xv, w1s[kk][tj * 4 + j], acc1[j]);
            }
        }
        __syncthreads();
    }
    T* o = (T*)a.out + (size_t)(slot0 + ts) * a.ldo;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int m = m0 + tj * 4 + j;
        if (m >= a.J) continue;
        if (MODE == 0) {
            const float wi = (a.in_wgt && my_pair >= 0) ? a.in_wgt[my_pair] : 1.f;
            const float g = acc0[j] * wi;
            o[m] = from_f32<T>(my_pair >= 0 ? g / (1.f + expf(-g)) * (acc1[j] * wi) : 0.f);
        } else if (MODE == 2) {
            const float r = fmaxf(acc0[j], 0.f);
            o[m] = from_f32<T>(my_pair >= 0 ? r * r : 0.f);
        } else {
            o[m] = from_f32<T>(acc0[j]);
        }
    }
}

extern "C" int braid_moe_gemm_simt(const void* x, const void* w0, const void* w1, void* out, const int* slot_pair,
                                   const int* tile_expert, const int* meta, int dtype, int mode, long long ldx,
                                   long long ldo, int J, int K, int top, int tile, int max_tiles, const float* in_wgt,
                                   long long w_expert, long long w_block, void* stream) {
    if (max_tiles <= 0 || J <= 0) return BRAID_OK;
    if (K <= 0) BRAID_REFUSE("moe_gemm: k=%d must be positive", K);
    if (tile <= 0 || tile % 16) BRAID_REFUSE("moe_gemm: the tile of %d slots must be a multiple of 16", tile);
    if (in_wgt && mode != 0) BRAID_REFUSE("moe_gemm: a weight on the expert's input goes with the gated first product (mode 0)");
    MoeGemmArgs a{x, w0, w1, out, slot_pair, tile_expert, meta, ldx, ldo, J, K, top, tile, in_wgt, w_expert, w_block};
    const long long units = (long long)max_tiles * (tile / 16);
    if (units > 65535) BRAID_REFUSE("moe_gemm: %lld units of 16 slots exceed the grid limit", units);
    dim3 grid((J + 63) / 64, (unsigned)units);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == BRAID_F32 && mode == 0) braid_launch(moe_gemm_simt_kernel<float, 0>, grid, dim3(256), 0, s, a);
    else if (dtype == BRAID_F32 && mode == 1) braid_launch(moe_gemm_simt_kernel<float, 1>, grid, dim3(256), 0, s, a);
    else if (dtype == BRAID_BF16 && mode == 0) braid_launch(moe_gemm_simt_kernel<__nv_bfloat16, 0>, grid, dim3(256), 0, s, a);
    else if (dtype == BRAID_BF16 && mode == 1) braid_launch(moe_gemm_simt_kernel<__nv_bfloat16, 1>, grid, dim3(256), 0, s, a);
    else if (dtype == BRAID_F32 && mode == 2) braid_launch(moe_gemm_simt_kernel<float, 2>, grid, dim3(256), 0, s, a);
    else if (dtype == BRAID_BF16 && mode == 2) braid_launch(moe_gemm_simt_kernel<__nv_bfloat16, 2>, grid, dim3(256), 0, s, a);
    else BRAID_REFUSE("moe_gemm: unknown dtype %d or mode %d", dtype, mode);
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ the experts' products on the tensor cores
// bfloat16, mma.sync with float32 accumulators (mma_tile.cuh).  One CTA a plan tile of BM slots (the plan's
// tile is BM) and BN outputs.  MODE 0 multiplies the gathered rows with the expert's gate and up matrices at
// once and stores silu(gate) * up; MODE 1 multiplies the activations with the down matrix; MODE 2 multiplies the
// gathered rows with the expert's up matrix alone and stores relu(.)^2.
template <int BM, int BN, int MODE>
__global__ void __launch_bounds__(128)
moe_gemm_mma_kernel(MoeGemmArgs a) {
    constexpr int NB = MODE == 0 ? 2 : 1;
    using Tile = MmaTile<BM, BN, (BM >= 64 ? 2 : 1), (BM >= 64 ? 2 : 4), NB>;
    extern __shared__ __align__(16) unsigned char moe_smem[];
    pdl_wait();
    const int t = blockIdx.y;
    if (t >= a.meta[0]) return;
    const int e = a.tile_expert[t];
    const int slot0 = t * BM, m0 = blockIdx.x * BN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int ACH = BM * 4 / 128 > 0 ? BM * 4 / 128 : 1;
    constexpr int BCH = BN * 4 / 128;
    const __nv_bfloat16* a_rows[ACH];
    const __nv_bfloat16* b_rows[NB][BCH];
    const __nv_bfloat16* x = (const __nv_bfloat16*)a.x;
#pragma unroll
    for (int i = 0; i < ACH; ++i) {
        const int r = (tid + i * 128) >> 2;
        a_rows[i] = nullptr;
        if (r < BM) {
            if (MODE != 1) {
                const int pair = a.slot_pair[slot0 + r];
                if (pair >= 0) a_rows[i] = x + (size_t)(pair / a.top) * a.ldx;
            } else {
                a_rows[i] = x + (size_t)(slot0 + r) * a.ldx;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < BCH; ++i) {
        const int m = m0 + ((tid + i * 128) >> 2);
        b_rows[0][i] = m < a.J ? moe_weight_row<__nv_bfloat16>(a, a.w0, e, m) : nullptr;
        if (MODE == 0) b_rows[NB - 1][i] = m < a.J ? moe_weight_row<__nv_bfloat16>(a, a.w1, e, m) : nullptr;
    }
    float acc[NB][Tile::MI][Tile::NI][4];
    Tile::run(acc, (__nv_bfloat16*)moe_smem, a_rows, b_rows, a.K, a.w0);
    // only here: a successor whose CTAs take their places while this kernel's are still spread unevenly over the SMs keeps
    // those places, and the weights it streams then come through few SMs (a decode step of 8 experts of width 4096: 1.80 ->
    // 1.42 ms)
    pdl_trigger();
    const int wm0 = (warp / (BM >= 64 ? 2 : 4)) * (BM / (BM >= 64 ? 2 : 1)), wn0 = (warp % (BM >= 64 ? 2 : 4)) * (BN / (BM >= 64 ? 2 : 4));
    __nv_bfloat16* out = (__nv_bfloat16*)a.out;
    const bool pairs_ok = (a.ldo & 1) == 0;
#pragma unroll
    for (int mi = 0; mi < Tile::MI; ++mi)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int slot = slot0 + wm0 + mi * 16 + (lane >> 2) + half * 8;
            const int pair_here = MODE == 1 ? 0 : a.slot_pair[slot];
            const bool live = pair_here >= 0;
            const float wi = (MODE == 0 && a.in_wgt && live) ? a.in_wgt[pair_here] : 1.f;
#pragma unroll
            for (int ni = 0; ni < Tile::NI; ++ni) {
                const int col = m0 + wn0 + ni * 8 + 2 * (lane & 3);
                float v0, v1;
                if (MODE == 0) {
                    const float g0 = acc[0][mi][ni][half * 2] * wi, g1 = acc[0][mi][ni][half * 2 + 1] * wi;
                    v0 = live ? g0 / (1.f + expf(-g0)) * (acc[NB - 1][mi][ni][half * 2] * wi) : 0.f;
                    v1 = live ? g1 / (1.f + expf(-g1)) * (acc[NB - 1][mi][ni][half * 2 + 1] * wi) : 0.f;
                } else if (MODE == 2) {
                    const float r0 = fmaxf(acc[0][mi][ni][half * 2], 0.f), r1 = fmaxf(acc[0][mi][ni][half * 2 + 1], 0.f);
                    v0 = live ? r0 * r0 : 0.f;
                    v1 = live ? r1 * r1 : 0.f;
                } else {
                    v0 = acc[0][mi][ni][half * 2];
                    v1 = acc[0][mi][ni][half * 2 + 1];
                }
                __nv_bfloat16* o = out + (size_t)slot * a.ldo + col;
                if (pairs_ok && col + 1 < a.J) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(v0, v1);
                else {
                    if (col < a.J) o[0] = __float2bfloat16_rn(v0);
                    if (col + 1 < a.J) o[1] = __float2bfloat16_rn(v1);
                }
            }
        }
}

extern "C" int braid_moe_gemm_mma(const void* x, const void* w0, const void* w1, void* out, const int* slot_pair,
                                  const int* tile_expert, const int* meta, int mode, long long ldx, long long ldo,
                                  int J, int K, int top, int tile, int max_tiles, const float* in_wgt, long long w_expert,
                                  long long w_block, void* stream) {
    if (max_tiles <= 0 || J <= 0) return BRAID_OK;
    if (K <= 0 || K % 8 || ldx % 8 || w_expert % 8 || w_block % 8) BRAID_REFUSE("moe_gemm_mma: k=%d, the row stride %lld and the weights' strides must be multiples of 8", K, ldx);
    if (((uintptr_t)x | (uintptr_t)w0 | (uintptr_t)w1) & 15) BRAID_REFUSE("moe_gemm_mma: operands must start on 16 bytes");
    if (tile != 16 && tile != 64) BRAID_REFUSE("moe_gemm_mma: the plan's tile must be 16 or 64 slots, not %d", tile);
    if (max_tiles > 65535) BRAID_REFUSE("moe_gemm_mma: %d tiles exceed the grid limit", max_tiles);
    if (in_wgt && mode != 0) BRAID_REFUSE("moe_gemm: a weight on the expert's input goes with the gated first product (mode 0)");
    MoeGemmArgs a{x, w0, w1, out, slot_pair, tile_expert, meta, ldx, ldo, J, K, top, tile, in_wgt, w_expert, w_block};
    cudaStream_t s = (cudaStream_t)stream;
    // the down product over tiles of 64 slots takes 128 outputs a CTA (its rows are fetched half as often: 0.36 -> 0.29 ms
    // at 2,048 tokens of width 2048); gate+up with its two accumulators stays at 64 (at 128 it needs 237 registers and
    // was 8 % slower), and so do tiles of 16
#define MOE_MMA(BM, BN, MODE)                                                                                   \
    do {                                                                                                        \
        using T_ = MmaTile<BM, BN, (BM >= 64 ? 2 : 1), (BM >= 64 ? 2 : 4), (MODE == 0 ? 2 : 1)>;                \
        static bool attr_set = false;                                                                           \
        if (!attr_set && T_::SMEM_BYTES > 48 * 1024) {                                                          \
            cudaError_t e_ = cudaFuncSetAttribute(moe_gemm_mma_kernel<BM, BN, MODE>,                            \
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, T_::SMEM_BYTES); \
            if (e_ != cudaSuccess) BRAID_REFUSE("moe_gemm_mma: shared memory: %s", cudaGetErrorString(e_));      \
            attr_set = true;                                                                                    \
        }                                                                                                       \
        braid_launch(moe_gemm_mma_kernel<BM, BN, MODE>, dim3((J + BN - 1) / BN, (unsigned)max_tiles), dim3(128), \
                     (size_t)T_::SMEM_BYTES, s, a);                                                             \
    } while (0)
    if (tile == 64 && mode == 0) MOE_MMA(64, 64, 0);
    else if (tile == 64 && mode == 1) MOE_MMA(64, 128, 1);
    else if (tile == 16 && mode == 0) MOE_MMA(16, 64, 0);
    else if (tile == 16 && mode == 1) MOE_MMA(16, 64, 1);
    else if (tile == 64 && mode == 2) MOE_MMA(64, 128, 2);
    else if (tile == 16 && mode == 2) MOE_MMA(16, 64, 2);
    else BRAID_REFUSE("moe_gemm_mma: unknown mode %d", mode);
#undef MOE_MMA
    BRAID_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ the weighted sum
// h[row, :] += sum over the row's choices k, in the order of k, of wgt[row, k] * y[pair_slot[row, k], :]
// (wgt null: every weight is 1, for experts whose weight went into their input).
// A thread owns V neighbouring columns of a row (16 bytes of y, or one number where sizes or starts do not allow that) and asks for
// up to MOE_COMBINE_BATCH choices' outputs at once; a CTA of 64 threads a span of columns, so that a decode step's few rows
// spread over the SMs.  12,288 outputs of 2,048 columns: 42 us with a CTA a row and 2-byte loads in a chain, 18 so; 8 rows of 6 choices
// 15 and 2.7 us.
#define MOE_COMBINE_THREADS 64
#define MOE_COMBINE_BATCH 8
template <typename T, int V>
__global__ void __launch_bounds__(MOE_COMBINE_THREADS)
moe_combine_kernel(float* __restrict__ h, const T* __restrict__ y, const int* __restrict__ pair_slot,
                   const float* __restrict__ wgt, int width, int top, long long ldy) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x, c = (blockIdx.y * MOE_COMBINE_THREADS + threadIdx.x) * V;
    if (c >= width) return;
    float* hr = h + (size_t)row * width + c;
    float old[V], acc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.f;
    if constexpr (V == 1) old[0] = hr[0];
    else
#pragma unroll
        for (int e = 0; e < V; e += 4) *reinterpret_cast<float4*>(old + e) = *reinterpret_cast<const float4*>(hr + e);
    for (int k0 = 0; k0 < top; k0 += MOE_COMBINE_BATCH) {
        int slot[MOE_COMBINE_BATCH];
        float w[MOE_COMBINE_BATCH], v[MOE_COMBINE_BATCH][V];
#pragma unroll
        for (int k = 0; k < MOE_COMBINE_BATCH; ++k) {
            slot[k] = k0 + k < top ? pair_slot[(size_t)row * top + k0 + k] : -1;
            w[k] = (wgt && k0 + k < top) ? wgt[(size_t)row * top + k0 + k] : 1.f;
        }
#pragma unroll
        for (int k = 0; k < MOE_COMBINE_BATCH; ++k)
            if (slot[k] >= 0) load_run<T, V>(y + (size_t)slot[k] * ldy + c, v[k]);
#pragma unroll
        for (int k = 0; k < MOE_COMBINE_BATCH; ++k)
            if (slot[k] >= 0)
#pragma unroll
                for (int e = 0; e < V; ++e) acc[e] = fmaf(w[k], v[k][e], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] += old[e];
    if constexpr (V == 1) hr[0] = acc[0];
    else
#pragma unroll
        for (int e = 0; e < V; e += 4) *reinterpret_cast<float4*>(hr + e) = *reinterpret_cast<const float4*>(acc + e);
}

template <typename T>
static void launch_moe_combine(float* h, const T* y, const int* pair_slot, const float* wgt, int rows, int width, int top, long long ldy,
                               cudaStream_t s) {
    constexpr int V = 16 / sizeof(T);
    const bool wide = width % V == 0 && ldy % V == 0 && (((uintptr_t)h | (uintptr_t)y) & 15) == 0;
    const int span = MOE_COMBINE_THREADS * (wide ? V : 1);
    const dim3 grid(rows, (width + span - 1) / span);
    if (wide) braid_launch(moe_combine_kernel<T, V>, grid, dim3(MOE_COMBINE_THREADS), 0, s, h, y, pair_slot, wgt, width, top, ldy);
    else braid_launch(moe_combine_kernel<T, 1>, grid, dim3(MOE_COMBINE_THREADS), 0, s, h, y, pair_slot, wgt, width, top, ldy);
}

extern "C" int braid_moe_combine(float* h, const void* y, int y_dtype, const int* pair_slot, const float* wgt,
                                 int rows, int width, int top, long long ldy, void* stream) {
    if (rows <= 0) return BRAID_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (width > 65535 * MOE_COMBINE_THREADS) BRAID_REFUSE("moe_combine: %d columns exceed one launch", width);
    if (y_dtype == BRAID_F32) launch_moe_combine(h, (const float*)y, pair_slot, wgt, rows, width, top, ldy, s);
    else if (y_dtype == BRAID_BF16) launch_moe_combine(h, (const __nv_bfloat16*)y, pair_slot, wgt, rows, width, top, ldy, s);
    else BRAID_REFUSE("moe_combine: unknown dtype code %d", y_dtype);
    BRAID_LAUNCH_CHECK();
}
