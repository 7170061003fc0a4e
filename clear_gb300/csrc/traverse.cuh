// Device-side ray/box and ray/triangle tests and node access, shared by the
// traversal kernels and the path tracer.  Every float operation is rounded
// separately (common.cuh), matching the reference's expressions.
#pragma once

#include "common.cuh"

namespace clr {

// Depth bound of the radix tree plus one (3b + 32 levels for b <= 21).
constexpr int kStackSize = 96;

struct Ray {
    float ox, oy, oz, tmax;
    float dx, dy, dz;
};

__device__ __forceinline__ Ray load_ray(const float4* rays, uint32_t r) {
    const float4 a = __ldg(rays + 2ull * r), b = __ldg(rays + 2ull * r + 1u);
    return Ray{a.x, a.y, a.z, a.w, b.x, b.y, b.z};
}

// rayAABBIntersection (OpenCL/bvh_traversal.cl:160-179), Woo's outside-plane
// test.  Returns the part of the test that does not depend on the bound;
// `entry` receives the entry distance maxt (-inf when the origin is inside),
// and the full test is  result && !(entry > tBound).
__device__ __forceinline__ bool box_test(float mnx, float mny, float mnz, float mxx, float mxy, float mxz,
                                         const Ray& r, float& entry) {
    const bool lx = r.ox < mnx, ux = r.ox > mxx;
    const bool ly = r.oy < mny, uy = r.oy > mxy;
    const bool lz = r.oz < mnz, uz = r.oz > mxz;
    if (!(lx | ux | ly | uy | lz | uz)) {
        entry = -INFINITY;
        return true;
    }
    const float cx = lx ? mnx : (ux ? mxx : 0.0f);
    const float cy = ly ? mny : (uy ? mxy : 0.0f);
    const float cz = lz ? mnz : (uz ? mxz : 0.0f);
    const float tx = ((lx | ux) && r.dx != 0.0f) ? fdiv(fsub(cx, r.ox), r.dx) : -1.0f;
    const float ty = ((ly | uy) && r.dy != 0.0f) ? fdiv(fsub(cy, r.oy), r.dy) : -1.0f;
    const float tz = ((lz | uz) && r.dz != 0.0f) ? fdiv(fsub(cz, r.oz), r.dz) : -1.0f;
    const float maxt = fmaxf(tx, fmaxf(ty, tz));
    entry = maxt;
    if (maxt < 0.0f) return false;
    const float qx = fadd(r.ox, fmul(maxt, r.dx));
    const float qy = fadd(r.oy, fmul(maxt, r.dy));
    const float qz = fadd(r.oz, fmul(maxt, r.dz));
    const bool hx = (qx >= mnx && qx <= mxx) || tx == maxt;
    const bool hy = (qy >= mny && qy <= mxy) || ty == maxt;
    const bool hz = (qz >= mnz && qz <= mxz) || tz == maxt;
    return hx && hy && hz;
}

// Same result as box_test, with fewer IEEE divisions: t = (plane - o) / d is
// first estimated with the ray's reciprocal direction; only axes whose
// estimate lies within 2^-20 (relative) of the largest estimate can hold the
// maximum, and only those are divided exactly.  An estimate is within a few
// ulp of the exact quotient, so every other axis is strictly below the exact
// maximum: its exact value would neither win the max nor satisfy t == maxt.
__device__ __forceinline__ bool box_test_fast(float mnx, float mny, float mnz, float mxx, float mxy, float mxz,
                                              const Ray& r, float ix, float iy, float iz, float& entry) {
    const bool lx = r.ox < mnx, ux = r.ox > mxx;
    const bool ly = r.oy < mny, uy = r.oy > mxy;
    const bool lz = r.oz < mnz, uz = r.oz > mxz;
    if (!(lx | ux | ly | uy | lz | uz)) {
        entry = -INFINITY;
        return true;
    }
    const float cx = lx ? mnx : (ux ? mxx : 0.0f);
    const float cy = ly ? mny : (uy ? mxy : 0.0f);
    const float cz = lz ? mnz : (uz ? mxz : 0.0f);
    const bool ax = (lx | ux) && r.dx != 0.0f;
    const bool ay = (ly | uy) && r.dy != 0.0f;
    const bool az = (lz | uz) && r.dz != 0.0f;
    float tx = ax ? (cx - r.ox) * ix : -1.0f;
    float ty = ay ? (cy - r.oy) * iy : -1.0f;
    float tz = az ? (cz - r.oz) * iz : -1.0f;
    const float m = fmaxf(tx, fmaxf(ty, tz));
    if (m < 0.0f) {  // every quotient is negative (signs are exact)
        entry = m;
        return false;
    }
    const float thr = (m < 3.0e38f) ? m - fabsf(m) * 0x1p-20f - 1e-30f : -INFINITY;
    if (ax && tx >= thr) tx = fdiv(fsub(cx, r.ox), r.dx);
    if (ay && ty >= thr) ty = fdiv(fsub(cy, r.oy), r.dy);
    if (az && tz >= thr) tz = fdiv(fsub(cz, r.oz), r.dz);
    const float maxt = fmaxf(tx, fmaxf(ty, tz));
    entry = maxt;
    if (maxt < 0.0f) return false;
    const float qx = fadd(r.ox, fmul(maxt, r.dx));
    const float qy = fadd(r.oy, fmul(maxt, r.dy));
    const float qz = fadd(r.oz, fmul(maxt, r.dz));
    const bool hx = (qx >= mnx && qx <= mxx) || tx == maxt;
    const bool hy = (qy >= mny && qy <= mxy) || ty == maxt;
    const bool hz = (qz >= mnz && qz <= mxz) || tz == maxt;
    return hx && hy && hz;
}

// rayTriangleIntersection (OpenCL/bvh_traversal.cl:54-108), Moller-Trumbore
// with |det| < 1e-6 rejected: whether the ray meets the triangle at some
// tt >= 0, and tt with its barycentrics, before any comparison with the
// current bound.  Record = {p0, id}, {p1-p0}, {p2-p0}.  One early exit only:
// the searches test with a few lanes of a warp, of which one usually passes, so
// five exits cost their branches (scattered rays 11.74 -> 11.32 ms, 64
// random-triangle scenes 57.6 -> 54.3); this one still pays where all lanes
// miss together (terrain render 41.3 -> 40.3).
__device__ __forceinline__ bool tri_eval(const float4 a, const float4 e1, const float4 e2, const Ray& r, float& tt,
                                         float& b1, float& b2) {
    const float px = fsub(fmul(r.dy, e2.z), fmul(r.dz, e2.y));
    const float py = fsub(fmul(r.dz, e2.x), fmul(r.dx, e2.z));
    const float pz = fsub(fmul(r.dx, e2.y), fmul(r.dy, e2.x));
    const float det = dot3(e1.x, e1.y, e1.z, px, py, pz);
    const bool flat = det > -0.000001f && det < 0.000001f;
    const float invDet = fdiv(1.0f, det);
    const float dx = fsub(r.ox, a.x), dy = fsub(r.oy, a.y), dz = fsub(r.oz, a.z);
    b1 = fmul(dot3(dx, dy, dz, px, py, pz), invDet);
    if (flat | (b1 < 0.0f) | (b1 > 1.0f)) return false;
    const float qx = fsub(fmul(dy, e1.z), fmul(dz, e1.y));
    const float qy = fsub(fmul(dz, e1.x), fmul(dx, e1.z));
    const float qz = fsub(fmul(dx, e1.y), fmul(dy, e1.x));
    b2 = fmul(dot3(r.dx, r.dy, r.dz, qx, qy, qz), invDet);
    tt = fmul(dot3(e2.x, e2.y, e2.z, qx, qy, qz), invDet);
    return !((b2 < 0.0f) | (fadd(b1, b2) > 1.0f) | (tt < 0.0f));
}

// The reference's test against the current bound t: a hit at tt > t is
// rejected (so an equal-t hit tested later wins), an accepted one moves t.
__device__ __forceinline__ bool tri_test(const float4 a, const float4 e1, const float4 e2, const Ray& r, float& t,
                                         float* b1_out = nullptr, float* b2_out = nullptr) {
    float tt, b1, b2;
    if (!tri_eval(a, e1, e2, r, tt, b1, b2) || tt > t) return false;
    t = tt;
    if (b1_out) *b1_out = b1;
    if (b2_out) *b2_out = b2;
    return true;
}

__device__ __forceinline__ bool tri_hit(const float4* __restrict__ tris, uint32_t leaf, const Ray& r, float& t,
                                        uint32_t& id) {
    const float4 a = __ldg(tris + 3u * leaf), b = __ldg(tris + 3u * leaf + 1u), c = __ldg(tris + 3u * leaf + 2u);
    if (tri_test(a, b, c, r, t)) {
        id = __float_as_uint(a.w);
        return true;
    }
    return false;
}

// ------------------------------------------------------ slab classification
//
// The searches need Woo's test (box_test) for two boxes per node, but its
// answer is almost always clear from the slab distances: per axis the two
// quotients (plane - o) / d are estimated as (plane - o) * (1 / d), lo <= hi,
// tn = the largest lo, tf = the smallest hi.  slab_test answers from those and
// leaves to box_test_fast only the boxes whose answer could depend on rounding,
// so the set of accepted boxes is box_test's.  The search loops issue
// instructions in half of their cycles with 10 of 32 lanes active; box_test_fast
// for both children costs about 180 instructions a node, its divisions behind
// divergent branches, this about 60 (1,000 rays on a 34,848-triangle mesh: 88
// -> 65 us a call from this and keeping the next node in a register alone).
// (fma(plane, 1 / d, -o / d) would save six of them, but its error is relative
// to |o / d| rather than to the distance: too much for the entry distances of
// rays nearly parallel to an axis.)
//
// With u = 2^-24 and 1 / d from rcp.approx (2u), an estimate is within 4u of
// the real quotient (relative; its sign is exact), box_test's quotients within
// 2u, and its point o + maxt d within u (2 |maxt d| + |o|) of the real one.
// Let M = max_k |o_k / d_k| over the nonzero d_k, mr = 2^-23 M + 1e-30, m = 2^-19 |tn|
// + mr = 32u |tn| + 2u M (the constant covers products that underflow), tn+ =
// max(tn, 0), and second = the larger of 0 and the second largest lo.  Then
//   tf - tn+ <= -m  either tf <= -m: the origin lies beyond a slab the ray moves
//                   away from; or tn - tf >= m: the point at maxt lies outside
//                   axis tf's slab by more than its rounding: box_test rejects;
//   tf - tn+ > m and |tn| - second > m
//                   either tn < -m and tf > m: the origin is inside all slabs,
//                   box_test accepts with entry -inf; or maxt is the quotient
//                   of tn's axis alone (the others lie below it by more than
//                   the errors, and it is within 6u of tn) and the point at
//                   maxt lies inside the other two slabs by more than its
//                   rounding: accepted;
// anything else is unsure: grazing and corner hits, flat boxes entered through
// their flat axis, origins on a plane.  (tn's own axis passes box_test by t ==
// maxt, so for tn > 0 the tf of the other two axes will do: slab_flat_hit, on
// the unsure boxes only, settles the flat ones -- 3.9 a ray in the Cornell box,
// 9.9 -> 9.4 ms a frame; in slab_test itself it costs the other scenes 3 %.)
//
// A zero component needs no margin: its 1 / d is infinite, so the axis gives lo
// = -inf, hi = inf where the origin lies between the planes (box_test's point
// keeps that coordinate, and the axis takes no part), both infinite with one
// sign where it does not (tf - tn+ = -inf <= -m, also where m is infinite with tn: a
// miss, as in box_test), and NaN where the origin is on a plane.  With that axis
// in M instead no box was sure, and rays parallel to an axis were up to 2.5 times
// slower than by box_test alone: before the classification / so / now, 4 Mi
// vertical rays on 2 Mi triangles of a terrain mesh, closest hit 5.8 / 8.5 / 4.3
// ms, shadow 4.4 / 7.7 / 4.1; an orthographic camera's 4.3 / 7.6 / 3.2 and 3.0 / 6.8 /
// 3.2.
// Components that are tiny but not zero keep their large M: within about 1e-5 of
// an axis most boxes are unsure (the vertical rays tilted by 1e-7: 6.0 / 8.4 / 8.4).
//
// NaN anywhere (min / max propagate it) and rays with a nonzero d outside [2^-40,
// 2^40] in magnitude or an infinite M (mr is NaN) fail both tests.  An estimate
// past the float range counts as larger than any finite one.
typedef unsigned long long f32x2;  // two packed floats, the lower one first

__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// A ray's constants for slab_test, packed as a node's planes are: a box is
// {min x, min y}, {min z, max x}, {max y, max z}.
struct SlabRay {
    f32x2 o_xy, o_zx, o_yz;     // -o
    f32x2 iv_xy, iv_zx, iv_yz;  // 1 / d
    float mr;                   // the part of the margins that does not depend on the box
};

__device__ __forceinline__ SlabRay make_slab_ray(const Ray& r) {
    const float ix = rcp_approx(r.dx), iy = rcp_approx(r.dy), iz = rcp_approx(r.dz);
    SlabRay k;
    k.o_xy = pack2(-r.ox, -r.oy);
    k.o_zx = pack2(-r.oz, -r.ox);
    k.o_yz = pack2(-r.oy, -r.oz);
    k.iv_xy = pack2(ix, iy);
    k.iv_zx = pack2(iz, ix);
    k.iv_yz = pack2(iy, iz);
    const float ax = r.dx == 0.0f ? 0.0f : fabsf(ix), ay = r.dy == 0.0f ? 0.0f : fabsf(iy),
                az = r.dz == 0.0f ? 0.0f : fabsf(iz);  // zero components take no part
    const float lo = min_nan(fabsf(ix), fabsf(iy), fabsf(iz)), hi = max_nan(ax, ay, az);
    const float M = max_nan(fabsf(r.ox) * ax, fabsf(r.oy) * ay, fabsf(r.oz) * az);
    k.mr = (hi <= 0x1p40f && lo >= 0x1p-40f && M < INFINITY) ? M * 0x1p-23f + 1e-30f : __int_as_float(0x7FFFFFFF);
    return k;
}

// The ray again (its tmax left out) from its slab form, which keeps the origin,
// and its direction.
__device__ __forceinline__ Ray slab_ray(const SlabRay& k, const float4 d) {
    float x, y, z;
    unpack2(k.o_xy, x, y);
    unpack2(k.o_zx, z, x);
    return Ray{-x, -y, -z, INFINITY, d.x, d.y, d.z};
}

enum : int { kBoxMiss = 0, kBoxHit = 1, kBoxUnsure = 2 };

// Classifies one box; `entry` is its entry distance for a hit: -inf inside
// the box, else tn (within 6u of box_test's) or, with `exact`, box_test's own.
template <class GetRay>
__device__ __forceinline__ int slab_test(f32x2 p0, f32x2 p1, f32x2 p2, const SlabRay& k, GetRay ray, bool exact,
                                         float& entry) {
    const f32x2 s0 = add2(p0, k.o_xy), s1 = add2(p1, k.o_zx), s2 = add2(p2, k.o_yz);
    float ax, ay, az, bx, by, bz;
    unpack2(mul2(s0, k.iv_xy), ax, ay);
    unpack2(mul2(s1, k.iv_zx), az, bx);
    unpack2(mul2(s2, k.iv_yz), by, bz);
    const float lx = min_nan(ax, bx), ly = min_nan(ay, by), lz = min_nan(az, bz);
    const float tf = min_nan(max_nan(ax, bx), max_nan(ay, by), max_nan(az, bz));
    const float lxy = max_nan(lx, ly);
    const float tn = max_nan(lxy, lz);
    const float second = max_nan(min_nan(lx, ly), min_nan(lxy, lz), 0.0f);
    const float m = __fmaf_rn(fabsf(tn), 0x1p-19f, k.mr);
    const float d = tf - max_nan(tn, 0.0f), g = fabsf(tn) - second;
    const bool miss = d <= -m;
    const bool hit = d > m && g > m;
    const bool inside = tn < 0.0f;
    entry = inside ? -INFINITY : tn;
    if (exact && hit && !inside) {
        // the quotient of tn's axis (alone: the other lo lie below tn - m)
        float nx, ny, nz, xx, xy, xz;
        unpack2(s0, nx, ny);
        unpack2(s1, nz, xx);
        unpack2(s2, xy, xz);
        const Ray r = ray();
        const bool isx = lx == tn, isy = ly == tn;
        const float num = isx ? (ax <= bx ? nx : xx) : isy ? (ay <= by ? ny : xy) : (az <= bz ? nz : xz);
        entry = fdiv(num, isx ? r.dx : isy ? r.dy : r.dz);
    }
    return miss ? kBoxMiss : hit ? kBoxHit : kBoxUnsure;
}

// An unsure box that is flat, or nearly, on tn's axis: the hit test of
// slab_test with the tf of the other two axes.
__device__ __forceinline__ bool slab_flat_hit(f32x2 p0, f32x2 p1, f32x2 p2, const SlabRay& k, float& entry) {
    float ax, ay, az, bx, by, bz;
    unpack2(mul2(add2(p0, k.o_xy), k.iv_xy), ax, ay);
    unpack2(mul2(add2(p1, k.o_zx), k.iv_zx), az, bx);
    unpack2(mul2(add2(p2, k.o_yz), k.iv_yz), by, bz);
    const float lx = min_nan(ax, bx), ly = min_nan(ay, by), lz = min_nan(az, bz);
    const float lxy = max_nan(lx, ly);
    const float tn = max_nan(lxy, lz);
    const float second = max_nan(min_nan(lx, ly), min_nan(lxy, lz), 0.0f);
    const float hx = lx == tn ? INFINITY : max_nan(ax, bx), hy = ly == tn ? INFINITY : max_nan(ay, by),
                hz = lz == tn ? INFINITY : max_nan(az, bz);
    const float m = __fmaf_rn(fabsf(tn), 0x1p-19f, k.mr);
    entry = tn;
    return tn - second > m && min_nan(hx, hy, hz) - tn > m;
}

struct Node {
    f32x2 b0[3], b1[3];
    uint32_t ref0, ref1;
};

// A 64-byte node as two 32-byte loads when the node array is 32-byte aligned
// (`wide`, the same for the whole launch), else as four 16-byte ones.
__device__ __forceinline__ Node load_node(const float4* __restrict__ nodes, uint32_t i, bool wide) {
    f32x2 q[8];
    const f32x2* p = reinterpret_cast<const f32x2*>(nodes + 4ull * i);
    if (wide) {
        asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(q[0]), "=l"(q[1]), "=l"(q[2]), "=l"(q[3]) : "l"(p));
        asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(q[4]), "=l"(q[5]), "=l"(q[6]), "=l"(q[7]) : "l"(p + 4));
    } else {
#pragma unroll
        for (int j = 0; j < 8; j += 2)
            asm volatile("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(q[j]), "=l"(q[j + 1]) : "l"(p + j));
    }
    Node nd;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        nd.b0[j] = q[j];
        nd.b1[j] = q[3 + j];
    }
    nd.ref0 = (uint32_t)q[6];
    nd.ref1 = (uint32_t)(q[6] >> 32);
    return nd;
}

__device__ __forceinline__ bool nodes_wide(const float4* nodes) {
    return (reinterpret_cast<uintptr_t>(nodes) & 31u) == 0u;
}

// slab_test's answer for a search that accepts no box entered past `tmax`
// (kBounded): an entry within its rounding of tmax counts as unsure.
__device__ __forceinline__ int slab_bounded(int c, float e, float tmax) {
    const float d = e * 0x1p-21f;  // more than the 6u of slab_test's entry
    return c != kBoxHit || e == -INFINITY || e <= tmax - d ? c : e > tmax + d ? (int)kBoxMiss : (int)kBoxUnsure;
}

// The answer for an unsure box.
template <bool kBounded, class GetRay>
__device__ __forceinline__ bool unsure_box(f32x2 p0, f32x2 p1, f32x2 p2, const SlabRay& k, GetRay ray, bool exact,
                                           float& e, float tmax) {
    if (!exact && !kBounded && slab_flat_hit(p0, p1, p2, k, e)) return true;
    float b[6], ix, iy, iz;
    unpack2(p0, b[0], b[1]);
    unpack2(p1, b[2], b[3]);
    unpack2(p2, b[4], b[5]);
    unpack2(k.iv_xy, ix, iy);
    unpack2(k.iv_yz, iy, iz);
    return box_test_fast(b[0], b[1], b[2], b[3], b[4], b[5], ray(), ix, iy, iz, e) && !(kBounded && e > tmax);
}

// Both child boxes of a node: bit 0 / 1 set when box_test accepts child 0 /
// 1, with their entry distances as slab_test gives them.  With kBounded a box
// entered past `tmax` is not accepted either.  Unsure boxes are settled one
// after the other, so that the code exists once.  `ray()` gives the ray
// itself, needed only there (and for exact entries): the searches that are
// short of registers load it again.
template <bool kBounded = false, class GetRay>
__device__ __forceinline__ uint32_t node_boxes(const Node& nd, const SlabRay& k, GetRay ray, bool exact, float& e0,
                                               float& e1, float tmax = INFINITY) {
    int c0 = slab_test(nd.b0[0], nd.b0[1], nd.b0[2], k, ray, exact, e0);
    int c1 = slab_test(nd.b1[0], nd.b1[1], nd.b1[2], k, ray, exact, e1);
    if (kBounded) {
        c0 = slab_bounded(c0, e0, tmax);
        c1 = slab_bounded(c1, e1, tmax);
    }
    uint32_t acc = (c0 == kBoxHit ? 1u : 0u) | (c1 == kBoxHit ? 2u : 0u);
    uint32_t todo = (c0 == kBoxUnsure ? 1u : 0u) | (c1 == kBoxUnsure ? 2u : 0u);
    while (todo) {
        const bool second = !(todo & 1u);
        f32x2 p[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) p[j] = second ? nd.b1[j] : nd.b0[j];
        float e;
        const bool ok = unsure_box<kBounded>(p[0], p[1], p[2], k, ray, exact, e, tmax);
        if (second) {
            e1 = e;
            acc |= ok ? 2u : 0u;
            todo = 0u;
        } else {
            e0 = e;
            acc |= ok ? 1u : 0u;
            todo &= 2u;
        }
    }
    return acc;
}

// node_boxes with exact entries, by box_test_fast alone.
__device__ __forceinline__ uint32_t node_boxes_woo(const Node& nd, const Ray& r, const SlabRay& k, float& e0, float& e1) {
    float a[6], b[6], ix, iy, iz;
    unpack2(k.iv_xy, ix, iy);
    unpack2(k.iv_yz, iy, iz);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        unpack2(nd.b0[j], a[2 * j], a[2 * j + 1]);
        unpack2(nd.b1[j], b[2 * j], b[2 * j + 1]);
    }
    return (box_test_fast(a[0], a[1], a[2], a[3], a[4], a[5], r, ix, iy, iz, e0) ? 1u : 0u) |
           (box_test_fast(b[0], b[1], b[2], b[3], b[4], b[5], r, ix, iy, iz, e1) ? 2u : 0u);
}

// The root's box (root_box of clr_bvh), as node_boxes.
template <bool kBounded = false, class GetRay>
__device__ __forceinline__ bool root_box_hit(const float* root_box, const SlabRay& k, GetRay ray, bool exact, float& e,
                                             float tmax = INFINITY) {
    const float* b = root_box;
    const f32x2 p0 = pack2(__ldg(b), __ldg(b + 1)), p1 = pack2(__ldg(b + 2), __ldg(b + 4)),
                p2 = pack2(__ldg(b + 5), __ldg(b + 6));
    int c = slab_test(p0, p1, p2, k, ray, exact, e);
    if (kBounded) c = slab_bounded(c, e, tmax);
    if (c == kBoxUnsure) return unsure_box<kBounded>(p0, p1, p2, k, ray, exact, e, tmax);
    return c == kBoxHit;
}

// ---------------------------------------------- nearer-first with replay
//
// The reference's closest-hit search (bvh_traversal.cl:182-215) visits the
// children of a node in a fixed order and keeps the LAST triangle accepted at
// the smallest t; which triangle that is, on ties and near-ties, depends on the
// visiting order.  The fast search visits the nearer child first and decides,
// per ray, whether its answer is necessarily the reference's; if not, the ray
// is searched again in the reference's order (a "replay").
//
// Notation for one ray: a candidate is a triangle whose Moller-Trumbore test
// passes with tt >= 0 and whose boxes, leaf box and ancestors, pass the part
// of Woo's test that does not depend on the bound; G(j) is the largest entry
// distance over candidate j's boxes.  Exact arithmetic gives G(j) <= tt(j);
// with rounding G(j) can exceed tt(j) by a few ulp ("inversion").
//
// The fast search culls a box when its entry distance exceeds the relaxed
// bound t + kReplayDelta (|t| + S) (S: the scene box's largest extent / 16),
// tests every leaf it reaches, and records
//   T, B      the smallest tt and the triangle that first reached it,
//   G(B)      the largest entry distance over B's boxes, which is its leaf
//             box's: an ancestor's entry that is >= 0 comes from an axis on
//             which the origin lies outside the ancestor's slab, hence outside
//             the leaf's slab on the same side with the leaf's plane no nearer,
//             and (plane - o) / d is monotone in the plane under rounding,
//   t2        the smallest tt of every other candidate it tested.
// With V = max(T, G(B)), the answer (T, B) is final unless
//   t2 <= V                                   (a tie or near-tie), or
//   G(B) > T + kReplayDelta / 4 (|T| + S)     (B's own boxes lie well past it).
// Proof sketch, assuming no inversion exceeds kReplayDelta / 4 (|tt| + S):
// every other candidate then has tt > V.  Tested ones by t2 > V.  A culled
// one lies under a box whose entry exceeded the relaxed bound of a t >= T, so
// its G > T + kReplayDelta (|T| + S) >= V + kReplayDelta / 4 (|V| + S) (as
// G(B) is within kReplayDelta / 4 (|T| + S) of T), and its tt > V by the
// inversion bound.  In the reference's search, before B is tested t holds
// only tt values > V >= every entry on B's path, so B is reached and
// accepted, and no later candidate (tt > V >= T) is; the reference returns
// (T, B) with the same barycentrics.  Inversions measured on the
// random-triangle, terrain and Cornell scenes stay below 2^-21 relative; the
// bound assumed is 2^-14.
constexpr float kReplayDelta = 0x1p-12f;

__device__ __forceinline__ float replay_scale(const float* root_box) {
    const float ex = __ldg(root_box + 4) - __ldg(root_box + 0), ey = __ldg(root_box + 5) - __ldg(root_box + 1),
                ez = __ldg(root_box + 6) - __ldg(root_box + 2);
    const float m = fmaxf(ex, fmaxf(ey, ez));
    return (m < INFINITY) ? m * 0.0625f : 0.0f;
}

// slab_test's entry distances are within 6u of box_test's: the searches keep
// the winner's leaf entry rounded up by this factor as G(B), which can only
// replay more rays.
constexpr float kEntryUp = 1.0f + 0x1p-20f;

__device__ __forceinline__ float relaxed_bound(float t, float S) { return t + kReplayDelta * (fabsf(t) + S); }

__device__ __forceinline__ bool needs_replay(float t, float gbest, float t2, float S) {
    const float V = fmaxf(t, gbest);
    return (t2 < INFINITY && t2 <= V) || (gbest > t + 0.25f * kReplayDelta * (fabsf(t) + S));
}

}  // namespace clr
