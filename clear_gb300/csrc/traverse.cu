// BVH traversal on sm_103a: closest-hit and shadow (any-hit) queries.
//
// The root node index is root_box[3] (bit pattern).  clr_trace_closest
// visits nodes in the reference's order (OpenCL/bvh_traversal.cl:182-215):
// pop a node, handle child 0 then child 1, a leaf child is box-tested and its
// triangle tested at once, an internal child is pushed (so child 1's subtree
// is explored before child 0's).  The reference tests a popped node's box
// against the current t; here both child boxes are tested when their parent
// is loaded (one 64-byte node fetch) and the entry distance rides on the
// stack, compared with t at pop time.  The bound-independent half of the test
// does not depend on t, so the set of boxes accepted, and with it the hit, is
// the reference's.
// clr_trace_closest_ordered visits the nearer child first and replays, in the
// reference's order, every ray whose answer could depend on the order
// (traverse.cuh): the same ids and distances, with far fewer nodes visited.
#include <algorithm>

#include "common.cuh"
#include "search.cuh"

CLR_DEFINE_STATUS_READER(traverse)

namespace clr {

// Blocks per SM (72, 64 and 64 registers).  Nearer first, 5 / 6 / 7 / 8 blocks:
// camera rays 1.22 / 1.09 / 1.03 / 1.27 ms, rays in origin order 11.9 / 10.9 /
// 10.3 / 13.0 ms (the cases in search.cuh).  Reference's order, 6 / 7 / 8 / 9
// blocks: 5.17 / 5.13 / 4.87 / 5.00 ms.  Any hit, 7 / 8 / 9 blocks: 6.35 / 6.09 /
// 6.53 ms.
constexpr int kNearerBlocks = 7, kReferenceBlocks = 8, kShadowBlocks = 8;

// Rays searched again in the reference's order, summed over launches
// (clr_trace_replays).
static __device__ unsigned long long g_replays = 0;

// A block's chunk of a ray list.  With `order`, the r-th ray searched is
// rays[order[r]] (results go to its own index): rays sorted by origin share
// the tree's nodes.
struct ListIo {
    static constexpr bool kLeaf = false, kOneTree = true, kReplayCall = true;
    static constexpr uint32_t kMark = 0xFFFFFFFEu;  // in hit_id until the second search; no triangle's id
    const float4* rays;
    const uint32_t* order;
    Tree one_tree;
    uint32_t* hit_id;
    float* hit_t;
    __device__ __forceinline__ bool begin(uint32_t i, uint32_t& q, Tree&) const {
        q = order ? __ldg(order + i) : i;
        return true;
    }
    __device__ __forceinline__ Ray ray(uint32_t q) const { return load_ray(rays, q); }
    __device__ __forceinline__ float4 dir(uint32_t q) const { return __ldg(rays + 2ull * q + 1u); }
    __device__ __forceinline__ void done(uint32_t q, const Tree&, float t, uint32_t best) const {
        hit_id[q] = best;
        hit_t[q] = t;
    }
    __device__ __forceinline__ void mark(uint32_t q) const { hit_id[q] = kMark; }
    __device__ __forceinline__ bool marked(uint32_t q) const { return hit_id[q] == kMark; }
};

// kFast: the nearer-first search with replay; otherwise the reference's order.
// Both give the reference's ids and distances.
template <bool kFast>
__global__ void __launch_bounds__(kSearchThreads, kFast ? kNearerBlocks : kReferenceBlocks) k_trace_closest(Tree tree,
                                                                                  const float4* __restrict__ rays,
                                                                                  uint32_t nr,
                                                                                  const uint32_t* __restrict__ order,
                                                                                  Spread sp, uint32_t* hit_id,
                                                                                  float* hit_t) {
    __shared__ ClosestShared sh;
    uint2 over[kStackSize - kSharedStack];
    search_init(sh);
    ListIo io{rays, order, tree, hit_id, hit_t};
    if (kFast) {
        const uint32_t replays = search_nearer(io, nr, sp, sh, over);
        if (replays) atomicAdd(&g_replays, (unsigned long long)replays);
    } else {
        search_reference<false>(io, nr, sp, sh, over);
    }
}

// Any-hit: the bound stays at tmax, so the accepted set of boxes does not
// depend on the visiting order; the first accepted triangle ends the query.
// kNearFirst searches the nearer child of a node first: a blocker is met
// sooner when the rays of a warp are close together (origin order).
template <bool kNearFirst>
__global__ void __launch_bounds__(kSearchThreads, kShadowBlocks) k_trace_shadow(Tree tree,
                                                                                const float4* __restrict__ rays,
                                                                                uint32_t nr,
                                                                                const uint32_t* __restrict__ order,
                                                                                Spread sp, uint8_t* __restrict__ occluded) {
    __shared__ uint32_t s_stack[kSharedStack * kSearchThreads];
    __shared__ uint32_t s_next;
    uint32_t over[kStackSize - kSharedStack];
    Stack<uint32_t> stack{s_stack + threadIdx.x, over, 0};
    const bool wide = nodes_wide(tree.nodes);
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    if (!spread_lane(sp)) return;
    SlabRay slab;
    float tmax;
    uint32_t cur, q, guard;
    bool occ;
    auto get_ray = [&]() { return load_ray(rays, q); };
    auto hit_leaf = [&](uint32_t ref) {
        float t = tmax;
        uint32_t id;
        return tri_hit(tree.tris, ref & ~kLeafBit, get_ray(), t, id);
    };
    auto begin = [&](uint32_t i) {
        q = order ? __ldg(order + i) : i;
        const Ray ray = get_ray();
        slab = make_slab_ray(ray);
        tmax = ray.tmax;
        cur = kNoNode;
        guard = 0;
        occ = false;
        float e;
        if (tree.n && root_box_hit<true>(tree.root_box, slab, get_ray, false, e, tmax)) {
            if (tree.n >= 2) cur = __float_as_uint(__ldg(tree.root_box + 3));
            else occ = hit_leaf(0u);
        }
    };
    uint64_t i = spread_ray(sp, atomicAdd(&s_next, 1u));
    if (i >= nr) return;
    begin((uint32_t)i);
    uint32_t pend = kNoNode;  // a leaf waiting for its test
    for (;;) {
        Node nd;
        const bool have = cur != kNoNode;
        if (have) nd = load_node(tree.nodes, cur, wide);
        if (pend != kNoNode) {
            occ = hit_leaf(pend);
            pend = kNoNode;
            if (occ) {
                cur = kNoNode;
                stack.sp = 0;
            }
        }
        if (cur != kNoNode) {
            float e0, e1;
            uint32_t acc = node_boxes<true>(nd, slab, get_ray, false, e0, e1, tmax);
            if (++guard >= tree.n) acc = stack.sp = 0;  // corrupt tree: a valid one has n - 1 nodes
            const bool both = acc == 3u, first1 = acc == 2u || (both && kNearFirst && e1 < e0);
            const uint32_t near = first1 ? nd.ref1 : nd.ref0, far = first1 ? nd.ref0 : nd.ref1;
            const bool nl = acc && (near & kLeafBit), fl = both && (far & kLeafBit);
            pend = nl ? near : fl ? far : kNoNode;
            cur = acc && !nl ? near : both && !fl ? far : kNoNode;
            if (both && nl == fl) stack.push(far);
        }
        if (cur == kNoNode && stack.sp > 0) {
            const uint32_t top = stack.pop();
            const bool leaf = (top & kLeafBit) != 0u;
            if (leaf && pend != kNoNode) {
                ++stack.sp;  // its turn comes after the waiting leaf's
            } else {
                cur = leaf ? kNoNode : top;
                pend = leaf ? top : pend;
            }
        }
        if (cur == kNoNode && pend == kNoNode) {
            occluded[q] = occ ? 1 : 0;
            i = spread_ray(sp, atomicAdd(&s_next, 1u));
            if (i >= nr) break;
            begin((uint32_t)i);
        }
    }
}

// Blocks of a search kernel that fit on the GPU at once.
template <typename K>
static unsigned int resident_blocks(K kernel) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSearchThreads, 0) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    return (unsigned int)(clr_sm_count() * per_sm);
}

}  // namespace clr

using namespace clr;

static int check_trace_args(const clr_bvh* bvh, const float* rays, uint32_t num_rays, const void* out0) {
    if (!bvh) return clr_set_error(CLR_EINVAL, "trace: bvh is NULL");
    if (num_rays == 0) return CLR_OK;
    if (!rays || !out0) return clr_set_error(CLR_EINVAL, "trace: NULL rays or output");
    if (reinterpret_cast<uintptr_t>(rays) & 15u) return clr_set_error(CLR_EINVAL, "trace: rays must be 16-byte aligned");
    if (bvh->num_tris > 0 && (!bvh->tris || !bvh->root_box || (bvh->num_tris > 1 && !bvh->nodes)))
        return clr_set_error(CLR_EINVAL, "trace: bvh buffers are NULL");
    return CLR_OK;
}

static Tree tree_of(const clr_bvh* bvh) {
    return Tree{static_cast<const float4*>(bvh->nodes), static_cast<const float4*>(bvh->tris), bvh->root_box,
                bvh->num_tris};
}

// Spread and grid of a ray list.  Above about 5 Mi triangles (560 MB of nodes and
// triangles) rays in no order suddenly pay far more for the same number of
// nodes: the reads reach past some cache of the memory path, at every ray count
// alike.  Rays that start together then do better than a pool that refills lane
// by lane, as they share what they read on the way down; so each chunk of 512
// rays is a block of its own, started by the hardware when one has ended.  4 Mi
// random rays, pool against this: 5 Mi triangles 7.9 / 6.9 ms, 8 Mi 11.2 / 8.8,
// 16 Mi 14.3 / 10.9 (shadow 7.7 / 7.2, 13.2 / 10.5, 18.5 / 14.4), but 4 Mi 5.7 /
// 6.2.  Chunks of 256 and 1,024 at 8 Mi: 8.9 and 9.3; half the blocks in flight:
// 11.1.  Rays sorted by origin do not meet that edge (5.3 / 6.3).
constexpr uint32_t kFarTreeTris = 5u << 20;
constexpr uint32_t kFarChunkShift = 9;

static unsigned int spread_list(uint32_t num_rays, uint32_t num_tris, bool sorted, unsigned int full, Spread& s) {
    const unsigned int grid = spread_for(num_rays, full, s);
    if (sorted || num_tris < kFarTreeTris || (num_rays >> kFarChunkShift) < full) return grid;
    s.shift = kFarChunkShift;
    return div_up(num_rays, 1u << kFarChunkShift);
}

template <bool kFast>
static int trace_closest(const clr_bvh* bvh, const float* rays, uint32_t num_rays, const uint32_t* order,
                         uint32_t* hit_id, float* hit_t, void* stream) {
    int rc = check_trace_args(bvh, rays, num_rays, hit_id);
    if (rc != CLR_OK || num_rays == 0) return rc;
    if (!hit_t) return clr_set_error(CLR_EINVAL, "clr_trace_closest: hit_t is NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto kernel = kFast && bvh->num_tris >= 2 ? k_trace_closest<true> : k_trace_closest<false>;  // 1: no order
    Spread sp;
    const unsigned int grid = spread_list(num_rays, bvh->num_tris, order != nullptr, resident_blocks(kernel), sp);
    kernel<<<grid, kSearchThreads, 0, st>>>(tree_of(bvh), reinterpret_cast<const float4*>(rays), num_rays, order, sp,
                                            hit_id, hit_t);
    CLR_LAUNCH_CHECK("k_trace_closest");
    return CLR_OK;
}

static int trace_shadow(const clr_bvh* bvh, const float* rays, uint32_t num_rays, const uint32_t* order,
                        uint8_t* occluded, void* stream) {
    int rc = check_trace_args(bvh, rays, num_rays, occluded);
    if (rc != CLR_OK || num_rays == 0) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    auto kernel = order ? k_trace_shadow<true> : k_trace_shadow<false>;
    Spread sp;
    const unsigned int grid = spread_list(num_rays, bvh->num_tris, order != nullptr, resident_blocks(kernel), sp);
    kernel<<<grid, kSearchThreads, 0, st>>>(tree_of(bvh), r4, num_rays, order, sp, occluded);
    CLR_LAUNCH_CHECK("k_trace_shadow");
    return CLR_OK;
}

// The searches over a ray order (lbvh_build.cu sorts the rays).
int clr_trace_closest_in_order(const clr_bvh* bvh, const float* rays, uint32_t num_rays, const uint32_t* order,
                               uint32_t* hit_id, float* hit_t, void* stream) {
    return trace_closest<true>(bvh, rays, num_rays, order, hit_id, hit_t, stream);
}
int clr_trace_shadow_in_order(const clr_bvh* bvh, const float* rays, uint32_t num_rays, const uint32_t* order,
                              uint8_t* occluded, void* stream) {
    return trace_shadow(bvh, rays, num_rays, order, occluded, stream);
}

extern "C" int clr_trace_closest(const clr_bvh* bvh, const float* rays, uint32_t num_rays, uint32_t* hit_id,
                                 float* hit_t, void* stream) {
    return trace_closest<false>(bvh, rays, num_rays, nullptr, hit_id, hit_t, stream);
}

extern "C" int clr_trace_closest_ordered(const clr_bvh* bvh, const float* rays, uint32_t num_rays, uint32_t* hit_id,
                                         float* hit_t, void* stream) {
    return trace_closest<true>(bvh, rays, num_rays, nullptr, hit_id, hit_t, stream);
}

extern "C" int clr_trace_replays(uint64_t* count, int clear) {
    if (!count) return clr_set_error(CLR_EINVAL, "clr_trace_replays: NULL count");
    unsigned long long v = 0;
    CLR_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_replays, sizeof(v)));
    if (clear) {
        const unsigned long long z = 0;
        CLR_CUDA_TRY(cudaMemcpyToSymbol(g_replays, &z, sizeof(z)));
    }
    *count = v;
    return CLR_OK;
}

extern "C" int clr_trace_shadow(const clr_bvh* bvh, const float* rays, uint32_t num_rays, uint8_t* occluded,
                                void* stream) {
    return trace_shadow(bvh, rays, num_rays, nullptr, occluded, stream);
}
