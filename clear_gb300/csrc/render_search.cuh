// The renderers' ray searches over block pools (search.cuh): closest hits of
// the extended paths and visibility of the next-event shadow rays.  For scenes
// without cutouts, nearer-first (CLR_RENDER_ORDERED); the others search ray by
// ray (render_common.cuh).
#pragma once

#include "render_common.cuh"
#include "search.cuh"

namespace clr {

__device__ __forceinline__ Tree tree_of(const DScene& sc) { return Tree{sc.nodes, sc.tris, sc.root_box, sc.num_tris}; }

// Spread for queues whose length only the device knows: the grid holds the
// blocks that fit at once, those without rays leave.  Path rays have little to
// share with their neighbours in the queue, so a queue that does not fill the
// lanes goes to all warps, four rays to a block at a time (Cornell, 65,536
// paths: 10.4 ms on all lanes, 9.6 in chunks of 64 on 18 lanes a warp; chunks
// of 4 / 8 / 16 / 32: 7.74 / 7.82 / 8.04 / 8.47 at a later step).
__device__ __forceinline__ Spread spread_queue(uint32_t n) {
    Spread s;
    s.lanes = min(32u, n / (gridDim.x * (kSearchThreads / 32)) + 1u);
    s.shift = s.lanes < 32u ? 2u : 6u;
    return s;
}

// Hit record {id, t, b1, b2} of the ray on the triangle at `leaf` (the same
// arithmetic as in the search), or a miss for kNoNode.
__device__ __forceinline__ float4 hit_record(const Tree& tree, uint32_t leaf, const Ray& ray) {
    if (leaf == kNoNode) return make_float4(__uint_as_float(kNone32), INFINITY, 0.f, 0.f);
    const float4 a = __ldg(tree.tris + 3u * leaf);
    float t, b1, b2;
    tri_eval(a, __ldg(tree.tris + 3u * leaf + 1u), __ldg(tree.tris + 3u * leaf + 2u), ray, t, b1, b2);
    return make_float4(a.w, t, b1, b2);
}
constexpr uint32_t kHitMark = 0xFFFFFFFEu;  // in a hit record until the second search; no leaf and no face

// ------------------------------------------------------------- visibility
//
// shadow_visible for many rays.  The reference searches the closest hit and
// compares its face with the light's (pathtracer.cl:119-122).  The light's
// triangle is known, so its distance T on the ray is computed first (the
// same arithmetic as the search's test of that triangle): a ray that misses
// it sees no light, and the search becomes an any-hit search below T.  With M
// = kReplayDelta (|T| + S), the relaxed bound T + M for culling, and the
// notation and the inversion bound of traverse.cuh:
//   another candidate at tt < T - M blocks the light: it is tested in the
//   reference's search, or culled by a bound below its own boxes' entries,
//   which are below T; either way the reference's closest hit is nearer than T;
//   no such candidate, the light's leaf reached, and not needs_replay(T, G,
//   t2) with t2 the nearest other candidate: the light is the closest hit, as
//   in the nearer-first search whose bound has come down to T;
//   anything else (the light's leaf not reached, a near tie) is searched again
//   in the reference's order.
// The bound is there from the start and the search ends at the first blocker
// (shadow kernel of the Cornell box at 65,536 paths: 92 -> 60 us).
// Environment rays (no light face) are blocked by any hit; an environment ray
// of a path that has met a lamp also sees the light when that lamp is the
// closest hit, so it is searched as the lamp's ray when it meets the lamp's
// triangle.

// Triangle `face` on the ray: its distance and an upper bound of its leaf
// box's entry distance (infinity where slab_test is not sure of the box).
__device__ __forceinline__ bool light_on_ray(const DScene& sc, uint32_t face, const Ray& ray, const SlabRay& slab,
                                             float& T, float& G) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(sc.faces + 56u * (size_t)face);
    const float4 p0 = __ldg(sc.vertices + __ldg(w)), p1 = __ldg(sc.vertices + __ldg(w + 1)),
                 p2 = __ldg(sc.vertices + __ldg(w + 2));
    const float4 e1 = make_float4(fsub(p1.x, p0.x), fsub(p1.y, p0.y), fsub(p1.z, p0.z), 0.f);
    const float4 e2 = make_float4(fsub(p2.x, p0.x), fsub(p2.y, p0.y), fsub(p2.z, p0.z), 0.f);
    float b1, b2;
    if (!tri_eval(p0, e1, e2, ray, T, b1, b2)) return false;
    const float mnx = fminf(p0.x, fminf(p1.x, p2.x)), mny = fminf(p0.y, fminf(p1.y, p2.y)),
                mnz = fminf(p0.z, fminf(p1.z, p2.z));
    const float mxx = fmaxf(p0.x, fmaxf(p1.x, p2.x)), mxy = fmaxf(p0.y, fmaxf(p1.y, p2.y)),
                mxz = fmaxf(p0.z, fmaxf(p1.z, p2.z));
    // an upper bound needs no classification: box_test's entry is the largest
    // quotient of an outside axis, within 6u of the largest lo (NaN where the
    // origin lies on a plane of an axis the ray is parallel to)
    auto get_ray = [&]() { return ray; };
    float e;
    slab_test(pack2(mnx, mny), pack2(mnz, mxx), pack2(mxy, mxz), slab, get_ray, false, e);
    G = slab.mr < INFINITY && e == e ? e * kEntryUp : INFINITY;
    return true;
}

struct VisibleShared {
    uint32_t stack[kSharedStack * kSearchThreads];
    uint32_t next, replays;
};

// The rays of a queue: begin / ray / mark / marked as in search.cuh, and
//   uint32_t light(uint32_t q)            the entry's shadow_light_word
//   const DScene& scene(uint32_t q)
//   void visible(uint32_t q, bool yes)
template <class Io>
struct ExactVisible {
    static constexpr bool kLeaf = false, kOneTree = Io::kOneTree;
    Io& io;
    Tree one_tree;
    __device__ __forceinline__ bool begin(uint32_t i, uint32_t& q, Tree& tree) { return io.begin(i, q, tree); }
    __device__ __forceinline__ Ray ray(uint32_t q) const { return io.ray(q); }
    __device__ __forceinline__ bool marked(uint32_t q) const { return io.marked(q); }
    __device__ __forceinline__ void done(uint32_t q, const Tree&, float, uint32_t best) {
        const uint32_t light = io.light(q);
        io.visible(q, (light & kEnvLightBit) ? best == kNoNode || best == (light & ~kEnvLightBit) : best == light);
    }
};

template <class Io>
__device__ __forceinline__ void search_visible(Io& io, uint32_t n, const Spread& sp, ClosestShared& sh, uint2* over) {
    Stack<uint32_t> stack{reinterpret_cast<uint32_t*>(sh.stack) + threadIdx.x, reinterpret_cast<uint32_t*>(over), 0};
    SlabRay slab;
    Tree ray_tree{};
    const Tree& tree = Io::kOneTree ? io.one_tree : ray_tree;
    bool wide = Io::kOneTree && nodes_wide(io.one_tree.nodes);
    float T = 0.f, tr = 0.f, near_t = 0.f, G = 0.f, t2 = 0.f;
    uint32_t face = kNoNode, cur = kNoNode, pend = kNoNode, q = 0, guard = 0, replays = 0;
    bool seen = false, blocked = false;
    auto get_ray = [&]() { return io.ray(q); };
    auto leaf_test = [&](uint32_t ref) {
        const uint32_t leaf = ref & ~kLeafBit;
        const float4 a = __ldg(tree.tris + 3u * leaf);
        float tt, b1, b2;
        if (!tri_eval(a, __ldg(tree.tris + 3u * leaf + 1u), __ldg(tree.tris + 3u * leaf + 2u), get_ray(), tt, b1, b2))
            return;
        if (face == kNoNode) blocked = true;
        else if (__float_as_uint(a.w) == face) seen = tt == T;
        else if (tt < near_t) blocked = true;
        else t2 = fminf(t2, tt);
    };
    auto next = [&]() {
        for (;;) {
            const uint64_t i = spread_ray(sp, atomicAdd(&sh.next, 1u));
            if (i >= n) return false;
            if (!io.begin((uint32_t)i, q, ray_tree)) continue;
            const Ray ray = io.ray(q);
            slab = make_slab_ray(ray);
            const uint32_t light = io.light(q);
            face = light == kNone32 ? kNoNode : (light & ~kEnvLightBit);
            if (face != kNoNode && !light_on_ray(io.scene(q), face, ray, slab, T, G)) {
                if (!(light & kEnvLightBit)) {
                    io.visible(q, false);
                    continue;
                }
                face = kNoNode;  // the lamp is not on the ray: visible if nothing is
            }
            if (!Io::kOneTree) wide = nodes_wide(tree.nodes);
            const float S = tree.n ? replay_scale(tree.root_box) : 0.f;
            if (face == kNoNode) T = INFINITY;
            tr = relaxed_bound(T, S);
            near_t = T - kReplayDelta * (fabsf(T) + S);
            t2 = INFINITY;
            guard = 0;
            seen = blocked = false;
            float e;
            if (tree.n && root_box_hit(tree.root_box, slab, get_ray, false, e) && !(e > tr)) {
                cur = __float_as_uint(__ldg(tree.root_box + 3));
                if (cur & kLeafBit) {  // one triangle
                    pend = cur;
                    cur = kNoNode;
                }
            }
            return true;
        }
    };
    bool active = spread_lane(sp) && next();
    while (active) {
        Node nd;
        const bool have = cur != kNoNode;
        if (have) nd = load_node(tree.nodes, cur, wide);
        if (pend != kNoNode) {
            leaf_test(pend);
            pend = kNoNode;
            if (blocked) {
                cur = kNoNode;
                stack.sp = 0;
            }
        }
        if (cur != kNoNode) {
            float e0, e1;
            uint32_t acc = node_boxes(nd, slab, get_ray, false, e0, e1);
            if (++guard >= tree.n) acc = stack.sp = 0;  // corrupt tree: a valid one has n - 1 nodes
            if (e0 > tr) acc &= 2u;
            if (e1 > tr) acc &= 1u;
            const bool both = acc == 3u, first1 = acc == 2u || (both && e1 < e0);
            const uint32_t near = first1 ? nd.ref1 : nd.ref0, far = first1 ? nd.ref0 : nd.ref1;
            const bool nl = acc && (near & kLeafBit), fl = both && (far & kLeafBit);
            pend = nl ? near : fl ? far : kNoNode;
            cur = acc && !nl ? near : both && !fl ? far : kNoNode;
            if (both && nl == fl) stack.push(far);
        }
        while (cur == kNoNode && stack.sp > 0) {
            const uint32_t top = stack.pop();
            const bool leaf = (top & kLeafBit) != 0u;
            if (leaf && pend != kNoNode) {
                ++stack.sp;  // its turn comes after the waiting leaf's
                break;
            }
            cur = leaf ? kNoNode : top;
            pend = leaf ? top : pend;
        }
        if (cur == kNoNode && pend == kNoNode) {
            const float S = tree.n ? replay_scale(tree.root_box) : 0.f;
            if (!blocked && face != kNoNode && (!seen || needs_replay(T, G, t2, S))) {
                ++replays;
                io.mark(q);
            } else {
                io.visible(q, !blocked);
            }
            active = next();
        }
    }
    if (replays) atomicAdd(&sh.replays, replays);
    __syncthreads();
    if (sh.replays) {  // the same for the whole block
        if (threadIdx.x == 0) sh.next = 0;
        __syncthreads();
        ExactVisible<Io> exact{io, tree};
        if constexpr (Io::kOneTree) exact.one_tree = io.one_tree;
        search_reference<true>(exact, n, sp, sh, over);
    }
}

// ------------------------------------------------------------- shading order
//
// The shade kernels wait for instructions as much as for data: a warp whose
// paths hit different kinds of materials runs the code of all of them with a
// few lanes each.  So queued paths are put in order of what they hit, within
// chunks of kBinChunk (a path's result does not depend on where it is shaded;
// chunks need no counts from other blocks).  Before and after: gradient step
// (eight materials of three kinds) 42.1 -> 32.4 ms, Cornell 7.76 -> 7.47, terrain
// 46.5 -> 45.4, 64 random-triangle scenes 66.5 -> 62.9.
constexpr int kBinChunk = 1024;
__device__ __forceinline__ uint32_t chunks_of(uint32_t n) { return n / kBinChunk + (n % kBinChunk != 0u); }

// 0 for an escaped path, else by the hit material's components.
__device__ __forceinline__ uint32_t shade_class(const DScene& sc, uint32_t id) {
    if (id == kNone32) return 0u;
    const uint32_t mat = __ldg(reinterpret_cast<const uint32_t*>(sc.faces + 56u * (size_t)id) + 13) & 0xFFFFu;
    const uint8_t* m = sc.materials + mat;
    const uint32_t num = m[0];
    if (num == 0) return 1u;  // the blob may end with the 8 bytes of its MaterialInfo
    const uint32_t first = m[8];  // the first element's id
    return num == 1 ? 2u + min(first, 1u) + (first == kBxNewWard ? 1u : 0u)
                    : 5u + (first == kBxDiffuse ? 0u : first == kBxAshS ? 1u : 2u);
}

// The entry of a queue of n, binned by bin_chunk, that thread i of the shading
// grid takes: the first warp's worth of every whole chunk, then the second one's
// and so on, so that the warps which run side by side are at about the same
// class and share its code in the instruction cache (the replay pass had 3 to 7
// of its 16 to 22 cycles an instruction in fetches).  Gradient step 32.5 -> 31.9
// ms, 64 random-triangle scenes 63.1 -> 61.2; slices of 128 entries 32.0 and
// 61.4, of 256 32.3 and 62.3.
constexpr uint32_t kBinSlice = 32;
__device__ __forceinline__ uint32_t binned_entry(uint32_t i, uint32_t n) {
    const uint32_t chunks = n / kBinChunk;
    if (i >= chunks * kBinChunk) return i;  // the last, partial chunk
    const uint32_t s = i / kBinSlice;
    return (s % chunks) * kBinChunk + (s / chunks) * kBinSlice + i % kBinSlice;
}

struct BinShared {
    uint32_t cnt[8][kBinChunk / 32];
    uint32_t base[2];
};

// This thread's place among the block's kBinChunk entries in order of their
// class (8: none), stable; afterwards sh.cnt[k][0] is where class k starts.
// The whole block enters, and calls __syncthreads() before it enters again.
__device__ __forceinline__ uint32_t bin_place(uint32_t cls, BinShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t rank = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const unsigned int m = __ballot_sync(0xFFFFFFFFu, cls == k);
        if (lane == 0) sh.cnt[k][warp] = __popc(m);
        if (cls == k) rank = __popc(m & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the 256 counts, eight per lane
        uint32_t v[8], sum = 0;
        uint32_t* c = &sh.cnt[0][0] + 8 * lane;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            v[k] = sum;
            sum += c[k];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = x - sum + v[k];
    }
    __syncthreads();
    return cls < 8u ? sh.cnt[cls][warp] + rank : 0u;
}

// Reorders queue[c0, c0 + kBinChunk) (of n entries in all) by class, in place.
template <class ClassOf>
__device__ __forceinline__ void bin_chunk(uint32_t* queue, uint32_t c0, uint32_t n, ClassOf class_of, BinShared& sh) {
    const uint32_t i = c0 + threadIdx.x;
    const uint32_t p = i < n ? queue[i] : 0u;
    const uint32_t at = bin_place(i < n ? class_of(p) : 8u, sh);
    if (i < n) queue[c0 + at] = p;
    __syncthreads();
}

}  // namespace clr
