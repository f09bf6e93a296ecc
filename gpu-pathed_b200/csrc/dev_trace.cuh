// Ray queries against the wide BVH: closest hit and any hit.
//
// Primitive tests restate the reference's arithmetic with uncontracted IEEE single
// operations (__fmul_rn/__fadd_rn/__fsub_rn/__fdiv_rn/__fsqrt_rn):
//   Triangle::hit  src/primitives/triangle.cu:7-48   (Moller-Trumbore form, inclusive bounds)
//   Sphere::hit    src/primitives/sphere.cu:7-43     (near root, then far root, strict bounds)
// and World::hit's selection rule (src/world.cu:5-41): a linear scan of all triangles in index
// order accepting t <= tNear (so on an exact tie the higher triangle index wins), then all
// spheres accepting only t < tNear (so triangles win ties against spheres and, among spheres,
// the lower index wins). Here the same outcome is computed as the minimum of a total order
// (t, then the tie rank), which does not depend on the order the BVH visits leaves in.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "dev_math.cuh"
#include "pt_types.h"

namespace pt {

// 32-byte loads and stores (one instruction and one full sector per lane on sm_100a; 32-byte
// aligned). The load names 64-bit elements: with v8.f32 ptxas 12.9 crashes on the shade kernels.
struct F8 {
    float4 a, b;
};
__device__ __forceinline__ F8 load8(const float4* p) {
    F8 v;
    double d0, d1, d2, d3;
    asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(d0), "=d"(d1), "=d"(d2), "=d"(d3) : "l"(p));
    v.a = make_float4(__int_as_float(__double2loint(d0)), __int_as_float(__double2hiint(d0)),
                      __int_as_float(__double2loint(d1)), __int_as_float(__double2hiint(d1)));
    v.b = make_float4(__int_as_float(__double2loint(d2)), __int_as_float(__double2hiint(d2)),
                      __int_as_float(__double2loint(d3)), __int_as_float(__double2hiint(d3)));
    return v;
}
__device__ __forceinline__ void store8(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

constexpr int kMissPrim = 0x7fffffff;  // no hit
// Relative slack applied to box-interval ends: boxes are visited when they might contain a
// hit the primitive test would accept (never culls what the linear scan reports).
constexpr float kBoxSlack = 1.00006103515625f;  // 1 + 2^-14

struct Hit {
    float t, b1, b2;
    int prim;  // >= 0 triangle id, < 0 ~sphere id, kMissPrim: none
};

__device__ __forceinline__ float xdot(V a, V b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ V xcross(V a, V b) {
    return V{__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)),
             -__fsub_rn(__fmul_rn(a.x, b.z), __fmul_rn(a.z, b.x)),
             __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x))};
}
__device__ __forceinline__ V xsub(V a, V b) {
    return V{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}

// Triangle::hit arithmetic. e1 = p1 - p0 and e2 = p2 - p0 arrive precomputed (same FP32
// subtractions). Returns false on a miss; otherwise t, b1, b2. tmax is inclusive.
__device__ __forceinline__ bool tri_test(V p0, V e1, V e2, V o, V d, float tmin, float tmax,
                                         float& t, float& b1, float& b2) {
    const V s1 = xcross(d, e2);
    const float divisor = xdot(s1, e1);
    if (divisor == 0.f) return false;
    const float inv = __fdiv_rn(1.f, divisor);
    const V s = xsub(o, p0);
    b1 = __fmul_rn(xdot(s, s1), inv);
    if (b1 < 0.f || b1 > 1.f) return false;
    const V s2 = xcross(s, e1);
    b2 = __fmul_rn(xdot(d, s2), inv);
    if (b2 < 0.f || __fadd_rn(b1, b2) > 1.f) return false;
    t = __fmul_rn(xdot(e2, s2), inv);
    if (t < tmin || t > tmax) return false;
    return true;
}

// Component k (0, 1, 2) of a vector, by selects (no local memory).
__device__ __forceinline__ float vcomp(V v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

// Watertight ray/triangle test (Woop, Benthin and Wald, "Watertight Ray/Triangle
// Intersection", JCGT 2(1), 2013), the opt-in alternative to Triangle::hit: no ray that
// passes through a shared edge or vertex of a closed mesh slips between its triangles.
// - Axes: kz is the largest component of |d| (first of x, y, z on ties), kx and ky the next two
//   cyclically, swapped when d[kz] < 0 so the winding is kept.
// - Shear: sz = 1 / d[kz], sx = d[kx] * sz, sy = d[ky] * sz (every operation rounded once).
// - Vertices relative to the origin, sheared so the ray runs along +z: ax = A[kx] - sx A[kz],
//   ay = A[ky] - sy A[kz] (likewise B, C).
// - Edge functions U = cx by - cy bx, V = ax cy - ay cx, W = bx ay - by ax; any that is exactly 0
//   is recomputed in FP64 from the same FP32 inputs (products exact, one rounding each).
// - Mixed signs miss; det = U + V + W, det = 0 misses; T = U sz A[kz] + V sz B[kz] + W sz C[kz],
//   t = T / det within [tmin, tmax] (inclusive, as Triangle::hit), b1 = V / det (weight of p1),
//   b2 = W / det (weight of p2). No backface culling, as the reference.
// Every FP32 operation is an explicit round-to-nearest intrinsic (no contraction), so the
// oracle's host restatement gives the same bits.
__device__ __forceinline__ bool tri_test_wt(V p0, V p1, V p2, V o, V d, float tmin, float tmax, float& t,
                                            float& b1, float& b2) {
    const float adx = fabsf(d.x), ady = fabsf(d.y), adz = fabsf(d.z);
    const int kz = adx >= ady ? (adx >= adz ? 0 : 2) : (ady >= adz ? 1 : 2);
    int kx = kz == 2 ? 0 : kz + 1;
    int ky = kx == 2 ? 0 : kx + 1;
    const float dz = vcomp(d, kz);
    if (dz < 0.f) {
        const int k = kx;
        kx = ky;
        ky = k;
    }
    const float sz = __fdiv_rn(1.f, dz);
    const float sx = __fmul_rn(vcomp(d, kx), sz), sy = __fmul_rn(vcomp(d, ky), sz);
    const V A = xsub(p0, o), B = xsub(p1, o), C = xsub(p2, o);
    const float Az = vcomp(A, kz), Bz = vcomp(B, kz), Cz = vcomp(C, kz);
    const float ax = __fsub_rn(vcomp(A, kx), __fmul_rn(sx, Az)), ay = __fsub_rn(vcomp(A, ky), __fmul_rn(sy, Az));
    const float bx = __fsub_rn(vcomp(B, kx), __fmul_rn(sx, Bz)), by = __fsub_rn(vcomp(B, ky), __fmul_rn(sy, Bz));
    const float cx = __fsub_rn(vcomp(C, kx), __fmul_rn(sx, Cz)), cy = __fsub_rn(vcomp(C, ky), __fmul_rn(sy, Cz));
    float U = __fsub_rn(__fmul_rn(cx, by), __fmul_rn(cy, bx));
    float Vv = __fsub_rn(__fmul_rn(ax, cy), __fmul_rn(ay, cx));
    float Ww = __fsub_rn(__fmul_rn(bx, ay), __fmul_rn(by, ax));
    if (U == 0.f || Vv == 0.f || Ww == 0.f) {
        U = __double2float_rn(__dsub_rn(__dmul_rn((double)cx, (double)by), __dmul_rn((double)cy, (double)bx)));
        Vv = __double2float_rn(__dsub_rn(__dmul_rn((double)ax, (double)cy), __dmul_rn((double)ay, (double)cx)));
        Ww = __double2float_rn(__dsub_rn(__dmul_rn((double)bx, (double)ay), __dmul_rn((double)by, (double)ax)));
    }
    if ((U < 0.f || Vv < 0.f || Ww < 0.f) && (U > 0.f || Vv > 0.f || Ww > 0.f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, Vv), Ww);
    if (det == 0.f) return false;
    const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, __fmul_rn(sz, Az)), __fmul_rn(Vv, __fmul_rn(sz, Bz))),
                              __fmul_rn(Ww, __fmul_rn(sz, Cz)));
    const float inv = __fdiv_rn(1.f, det);
    t = __fmul_rn(T, inv);
    if (!(t >= tmin && t <= tmax)) return false;
    b1 = __fmul_rn(Vv, inv);
    b2 = __fmul_rn(Ww, inv);
    return true;
}

// Sphere::hit root selection: the near root when it lies above tmin, else the far root.
// Returns false when neither root is above tmin (the caller applies the strict upper bound).
__device__ __forceinline__ bool sphere_candidate(V c, float r, V o, V d, float tmin, float& t) {
    const V oc = xsub(o, c);
    const float a = xdot(d, d);
    const float b = xdot(oc, d);
    const float cc = __fsub_rn(xdot(oc, oc), __fmul_rn(r, r));
    const float disc = __fsub_rn(__fmul_rn(b, b), __fmul_rn(a, cc));
    if (!(disc > 0.f)) return false;
    const float sq = __fsqrt_rn(disc);
    const float nb = -b;
    float tt = __fdiv_rn(__fsub_rn(nb, sq), a);
    if (tt > tmin) { t = tt; return true; }
    tt = __fdiv_rn(__fadd_rn(nb, sq), a);
    if (tt > tmin) { t = tt; return true; }
    return false;
}

struct RayPre {
    V o, d;
    float ix, iy, iz, ox, oy, oz;
};
__device__ __forceinline__ RayPre make_raypre(V o, V d) {
    RayPre r;
    r.o = o;
    r.d = d;
    const float dx = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
    const float dy = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
    const float dz = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
    r.ix = 1.f / dx;
    r.iy = 1.f / dy;
    r.iz = 1.f / dz;
    r.ox = o.x * r.ix;
    r.oy = o.y * r.iy;
    r.oz = o.z * r.iz;
    return r;
}

// Three-input min and max (one instruction on sm_100a); like fminf / fmaxf, a NaN input is ignored.
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Slab test of a box clipped to [tmin, tlim]: the entry distance, or +inf when the interval is
// empty (the box is visited when its entry tn and exit tf satisfy tn <= tf * kBoxSlack).
__device__ __forceinline__ float box_entry(const RayPre& r, float lx, float hx, float ly, float hy,
                                           float lz, float hz, float tmin, float tlim) {
    const float t0x = fmaf(lx, r.ix, -r.ox), t1x = fmaf(hx, r.ix, -r.ox);
    const float t0y = fmaf(ly, r.iy, -r.oy), t1y = fmaf(hy, r.iy, -r.oy);
    const float t0z = fmaf(lz, r.iz, -r.oz), t1z = fmaf(hz, r.iz, -r.oz);
    const float tn = max3(fminf(t0x, t1x), fminf(t0y, t1y), fmaxf(fminf(t0z, t1z), tmin));
    const float tf = min3(fmaxf(t0x, t1x), fmaxf(t0y, t1y), fminf(fmaxf(t0z, t1z), tlim));
    return (tn <= tf * kBoxSlack) ? tn : __int_as_float(0x7f800000);
}

// Compare-exchange of two children by entry distance (misses are +inf).
__device__ __forceinline__ void child_order(float& ta, int& ca, float& tb, int& cb) {
    const bool swap = tb < ta;
    const float t = swap ? ta : tb;
    const int c = swap ? ca : cb;
    ta = swap ? tb : ta;
    ca = swap ? cb : ca;
    tb = t;
    cb = c;
}
// Children sorted nearest first by size-optimal sorting networks (1, 5 and 19 comparators; Knuth,
// TAOCP vol. 3, 5.3.4).
template <int W>
__device__ __forceinline__ void sort_children(float (&t)[W], int (&c)[W]) {
    auto o = [&](int a, int b) { child_order(t[a], c[a], t[b], c[b]); };
    if constexpr (W == 2) {
        o(0, 1);
    } else if constexpr (W == 4) {
        o(0, 1); o(2, 3); o(0, 2); o(1, 3); o(1, 2);
    } else {
        static_assert(W == 8, "BVH width 2, 4 or 8");
        o(0, 2); o(1, 3); o(4, 6); o(5, 7); o(0, 4); o(1, 5); o(2, 6); o(3, 7); o(0, 1); o(2, 3); o(4, 5); o(6, 7);
        o(2, 4); o(3, 5); o(1, 4); o(3, 6); o(1, 2); o(3, 4); o(5, 6);
    }
}

// Closest-hit acceptance for one leaf entry (tie rules above). `tcur` is best.t or tmax.
// `wt`: the scene's triangle entries hold p0, p1, p2 and take the watertight test.
__device__ __forceinline__ void leaf_entry(const float4* __restrict__ prims, int e, const RayPre& r,
                                           float tmin, float tmax, Hit& best, bool wt) {
    const float4 a = __ldg(prims + 3 * e);
    const int id = __float_as_int(a.w);
    const float tcur = best.prim == kMissPrim ? tmax : best.t;
    if (id >= 0) {
        const float4 b = __ldg(prims + 3 * e + 1);
        const float4 c = __ldg(prims + 3 * e + 2);
        float t, b1, b2;
        const bool h = wt ? tri_test_wt(mkv(a), mkv(b), mkv(c), r.o, r.d, tmin, tcur, t, b1, b2)
                          : tri_test(mkv(a), mkv(b), mkv(c), r.o, r.d, tmin, tcur, t, b1, b2);
        if (h) {
            // equal t: the higher triangle index wins; a triangle beats a sphere
            if (t == tcur && best.prim != kMissPrim && best.prim >= 0 && id < best.prim) return;
            best.t = t;
            best.b1 = b1;
            best.b2 = b2;
            best.prim = id;
        }
    } else {
        const float4 b = __ldg(prims + 3 * e + 1);
        float t;
        if (sphere_candidate(mkv(a), b.x, r.o, r.d, tmin, t)) {
            const bool better = t < tcur ||
                                (t == tcur && best.prim != kMissPrim && best.prim < 0 && id > best.prim);
            // id = ~k: a larger id is a lower sphere index k
            if (better) {
                best.t = t;
                best.b1 = 0.f;
                best.b2 = 0.f;
                best.prim = id;
            }
        }
    }
}

// Any-hit acceptance for one leaf entry: true if the entry blocks [tmin, tmax].
__device__ __forceinline__ bool leaf_entry_any(const float4* __restrict__ prims, int e, const RayPre& r,
                                               float tmin, float tmax, bool wt) {
    const float4 a = __ldg(prims + 3 * e);
    const int id = __float_as_int(a.w);
    if (id >= 0) {
        const float4 b = __ldg(prims + 3 * e + 1);
        const float4 c = __ldg(prims + 3 * e + 2);
        float t, b1, b2;
        return wt ? tri_test_wt(mkv(a), mkv(b), mkv(c), r.o, r.d, tmin, tmax, t, b1, b2)
                  : tri_test(mkv(a), mkv(b), mkv(c), r.o, r.d, tmin, tmax, t, b1, b2);
    }
    const float4 b = __ldg(prims + 3 * e + 1);
    float t;
    return sphere_candidate(mkv(a), b.x, r.o, r.d, tmin, t) && t < tmax;
}

template <int W>
struct NodeView {
    float lo_x[W], hi_x[W], lo_y[W], hi_y[W], lo_z[W], hi_z[W];
    int child[W];
};

template <int W>
__device__ __forceinline__ void load_node(const float4* __restrict__ p, NodeView<W>& nv) {
    constexpr int kUsed = (7 * W + 3) / 4;  // float4s that hold bounds + children
    float4 raw[kUsed];
#pragma unroll
    for (int i = 0; i < kUsed; i++) raw[i] = __ldg(p + i);
    const float* f = reinterpret_cast<const float*>(raw);
#pragma unroll
    for (int k = 0; k < W; k++) {
        nv.lo_x[k] = f[0 * W + k];
        nv.hi_x[k] = f[1 * W + k];
        nv.lo_y[k] = f[2 * W + k];
        nv.hi_y[k] = f[3 * W + k];
        nv.lo_z[k] = f[4 * W + k];
        nv.hi_z[k] = f[5 * W + k];
        nv.child[k] = __float_as_int(f[6 * W + k]);
    }
}

// A float node (W = 4 or 8) read in the ray's octant order: per axis the near planes (the
// lower bounds where the ray's direction component is positive, the upper ones where it is
// negative) into lo_*, the far planes into hi_*. For a box with lower <= upper bound, the near
// plane's slab distance is the smaller one (fmaf is monotone in its first operand for a fixed
// nonzero factor), so the slab test needs no min/max per axis and gives the same entry and exit
// distances bit for bit. The choice of plane is an address offset per load.
template <int W>
__device__ __forceinline__ void load_node_oct(const float4* __restrict__ p, const RayPre& r, NodeView<W>& nv) {
    static_assert(W == 4 || W == 8, "octant loads need whole float4 planes");
    constexpr int A = W / 4;  // float4s per plane
    const int sx = __float_as_int(r.ix) < 0 ? A : 0;
    const int sy = __float_as_int(r.iy) < 0 ? A : 0;
    const int sz = __float_as_int(r.iz) < 0 ? A : 0;
    float4 raw[7 * A];
#pragma unroll
    for (int a = 0; a < A; a++) {
        raw[0 * A + a] = __ldg(p + 0 * A + sx + a);
        raw[1 * A + a] = __ldg(p + 1 * A - sx + a);
        raw[2 * A + a] = __ldg(p + 2 * A + sy + a);
        raw[3 * A + a] = __ldg(p + 3 * A - sy + a);
        raw[4 * A + a] = __ldg(p + 4 * A + sz + a);
        raw[5 * A + a] = __ldg(p + 5 * A - sz + a);
        raw[6 * A + a] = __ldg(p + 6 * A + a);
    }
    const float* f = reinterpret_cast<const float*>(raw);
#pragma unroll
    for (int k = 0; k < W; k++) {
        nv.lo_x[k] = f[0 * W + k];
        nv.hi_x[k] = f[1 * W + k];
        nv.lo_y[k] = f[2 * W + k];
        nv.hi_y[k] = f[3 * W + k];
        nv.lo_z[k] = f[4 * W + k];
        nv.hi_z[k] = f[5 * W + k];
        nv.child[k] = __float_as_int(f[6 * W + k]);
    }
}

// Slab test on near and far planes (load_node_oct): the entry distance, or +inf when empty.
__device__ __forceinline__ float box_entry_nf(const RayPre& r, float nx, float fx, float ny, float fy, float nz,
                                              float fz, float tmin, float tlim) {
    const float tnx = fmaf(nx, r.ix, -r.ox), tfx = fmaf(fx, r.ix, -r.ox);
    const float tny = fmaf(ny, r.iy, -r.oy), tfy = fmaf(fy, r.iy, -r.oy);
    const float tnz = fmaf(nz, r.iz, -r.oz), tfz = fmaf(fz, r.iz, -r.oz);
    const float tn = max3(tnx, tny, fmaxf(tnz, tmin));
    const float tf = min3(tfx, tfy, fminf(tfz, tlim));
    return (tn <= tf * kBoxSlack) ? tn : __int_as_float(0x7f800000);
}

// Scale of a quantized node's axis: the FP32 power of two with biased exponent e.
__device__ __forceinline__ float qscale(uint32_t e) { return __uint_as_float((e & 0xFFu) << 23); }


// A quantized node (qnode_bytes(W) bytes, W = 4 or 8) decoded into the float view: each plane
// is fmaf(q, scale, origin), which contains the float box the build quantized.
template <int W>
__device__ __forceinline__ void load_qnode(const float4* __restrict__ p, NodeView<W>& nv) {
    constexpr int kF4 = qnode_bytes(W) / 16;
    float4 raw[kF4];
#pragma unroll
    for (int i = 0; i < kF4; i++) raw[i] = __ldg(p + i);
    const uint32_t e = __float_as_uint(raw[0].w);
    const float ox = raw[0].x, oy = raw[0].y, oz = raw[0].z;
    const float sx = qscale(e), sy = qscale(e >> 8), sz = qscale(e >> 16);
    const uint32_t* u = reinterpret_cast<const uint32_t*>(raw);
    auto q = [&](int a, int k) { return (float)((u[4 + (a * W + k) / 4] >> (8 * ((a * W + k) & 3))) & 0xFFu); };
#pragma unroll
    for (int k = 0; k < W; k++) {
        nv.lo_x[k] = __fmaf_rn(q(0, k), sx, ox);
        nv.hi_x[k] = __fmaf_rn(q(1, k), sx, ox);
        nv.lo_y[k] = __fmaf_rn(q(2, k), sy, oy);
        nv.hi_y[k] = __fmaf_rn(q(3, k), sy, oy);
        nv.lo_z[k] = __fmaf_rn(q(4, k), sz, oz);
        nv.hi_z[k] = __fmaf_rn(q(5, k), sz, oz);
        nv.child[k] = (int)u[qnode_child_offset(W) / 4 + k];
    }
}

// Per-query work counters (only maintained when the CNT template flag is set).
struct TraceWork {
    unsigned nodes = 0;  // wide nodes loaded
    unsigned prims = 0;  // leaf entries tested
};

// The traversal stack of one lane: children still to visit, each with its entry distance
// (closest hit; an any-hit entry is the child alone), farthest at the bottom. The first
// `shared` entries of every lane lie in shared memory ([entry][thread]), deeper ones, which few
// lanes reach, in global memory. An entry carries all that its later visit needs: popping a child
// and culling it against the current hit reads no node. (The stack before held one entry per tree
// level, the parent and the slots left, and read a popped child's six planes from its parent
// again: seven dependent loads and a slab test per pop.) With it the node visit sorts (distance,
// child) pairs and stores them as they are. Warp instructions of a mesh launch 234M -> 184M; frames, before -> after:
// mesh 30.2 -> 27.6 ms, slit room 81.8 -> 75.7, Cornell 3.26 -> 3.10, spheres 25.9 -> 25.4.
template <bool ANY>
struct LaneStack {
    using Entry = std::conditional_t<ANY, int, int2>;
    Entry* s;         // this lane's first entry in shared memory
    int stride;       // entries between a lane's consecutive shared entries
    StackShape shape;
    __device__ __forceinline__ Entry* slot(int i) const {
        if (i < shape.shared) return s + i * stride;
        return reinterpret_cast<Entry*>(shape.spill) + (size_t)(i - shape.shared) * shape.spill_stride +
               (blockIdx.x * blockDim.x + threadIdx.x);
    }
    static __device__ __forceinline__ Entry entry(int child, float t) {
        if constexpr (ANY) return child;
        else return make_int2(child, __float_as_int(t));
    }
};

// Next child to visit, or kEmptyChild when the stack is empty. Closest hit: children that begin
// beyond the current hit are dropped (the slab test's own rule, with the bound of now; a NaN bound
// drops none). So are empty children: a ray whose direction is NaN or infinite on all axes finds
// every slab open, an empty child's too.
template <bool ANY>
__device__ __forceinline__ int stack_pop(const LaneStack<ANY>& st, float tmax, const Hit& best, int& sp,
                                         int bottom = 0) {
    if constexpr (ANY) {
        if (sp == bottom) return kEmptyChild;
        sp--;
        return *st.slot(sp);
    } else {
        const float thr = (best.prim == kMissPrim ? tmax : best.t) * kBoxSlack * kBoxSlack;
        while (sp > bottom) {
            sp--;
            const int2 e = *st.slot(sp);
            if (!(__int_as_float(e.y) > thr) && e.x != kEmptyChild) return e.x;
        }
        return kEmptyChild;
    }
}

// One internal-node visit of a live query (`cur` >= 0): test the node's children, push the
// farther hits (nearest on top for closest hit; for any hit, nearest on top with `near`, else in
// the node's order), descend into the first, or pop the stack when none was hit. The query ends
// (`alive` false) when the stack runs empty, or gives up with `overflow` set when it would exceed
// the stack's entries.
template <int W, bool ANY, bool CNT>
__device__ __forceinline__ void node_step(const float4* __restrict__ nodes, bool quant, const RayPre& r, float tmin,
                                          float tmax, const LaneStack<ANY>& st, const Hit& best, int& cur, int& sp,
                                          bool& alive, int& overflow, TraceWork* work, bool near = false,
                                          int bottom = 0) {
    constexpr int kNF4 = sizeof(BvhNode<W>) / 16;
    const float inf = __int_as_float(0x7f800000);
    NodeView<W> nv;
    // Float nodes are read in octant order (near, far planes): no min/max per axis. For any hit too since
    // the stack's entries left room for the plane offsets (shadow stage of the slit room 16.7 -> 14.4 ms).
    constexpr bool kOct = W >= 4;
    if (quant) load_qnode<W>(nodes + (size_t)cur * (qnode_bytes(W) / 16), nv);
    else if constexpr (kOct) load_node_oct<W>(nodes + (size_t)cur * kNF4, r, nv);
    else load_node<W>(nodes + (size_t)cur * kNF4, nv);
    if (CNT) work->nodes++;
    const float tcur = best.prim == kMissPrim ? tmax : best.t;
    const float tlim = tcur * kBoxSlack;
    float te[W];
#pragma unroll
    for (int k = 0; k < W; k++) {
        if (kOct && !quant) {  // an empty child's planes are inverted (+inf, -inf): it misses (or see stack_pop)
            te[k] = box_entry_nf(r, nv.lo_x[k], nv.hi_x[k], nv.lo_y[k], nv.hi_y[k], nv.lo_z[k], nv.hi_z[k], tmin, tlim);
        } else {
            te[k] = box_entry(r, nv.lo_x[k], nv.hi_x[k], nv.lo_y[k], nv.hi_y[k], nv.lo_z[k], nv.hi_z[k], tmin, tlim);
            if (nv.child[k] == kEmptyChild) te[k] = inf;
        }
    }
    if (!ANY || near) sort_children<W>(te, nv.child);
    // the hit children, farthest first (any hit: the node's last first): all but the last one, which
    // is visited now, go on the stack
    if constexpr (!ANY) {
        int next = te[0] == inf ? kEmptyChild : nv.child[0];  // sorted: the nearest
        if (sp + W - 1 <= st.shape.shared) {
            typename LaneStack<ANY>::Entry* top = st.s + sp * st.stride;
#pragma unroll
            for (int k = W - 1; k >= 1; k--)
                if (te[k] != inf) {
                    *top = LaneStack<ANY>::entry(nv.child[k], te[k]);
                    top += st.stride;
                    sp++;
                }
        } else {
#pragma unroll
            for (int k = W - 1; k >= 1; k--)
                if (te[k] != inf) *st.slot(sp++) = LaneStack<ANY>::entry(nv.child[k], te[k]);
        }
        if (sp > st.shape.cap) {
            overflow = 1;
            alive = false;  // reported to the host; the query gives up
        } else if (next == kEmptyChild) {
            next = stack_pop<ANY>(st, tmax, best, sp, bottom);
            if (next == kEmptyChild) alive = false;
        }
        cur = next;
        return;
    }
    int next = kEmptyChild;
    float tnext = 0.f;
    if (sp + W - 1 <= st.shape.shared) {
        typename LaneStack<ANY>::Entry* top = st.s + sp * st.stride;
#pragma unroll
        for (int k = W - 1; k >= 0; k--) {
            if (te[k] == inf) continue;
            if (next != kEmptyChild) {
                *top = LaneStack<ANY>::entry(next, tnext);
                top += st.stride;
                sp++;
            }
            next = nv.child[k];
            tnext = te[k];
        }
    } else {
#pragma unroll
        for (int k = W - 1; k >= 0; k--) {
            if (te[k] == inf) continue;
            if (next != kEmptyChild) *st.slot(sp++) = LaneStack<ANY>::entry(next, tnext);
            next = nv.child[k];
            tnext = te[k];
        }
    }
    if (sp > st.shape.cap) {
        overflow = 1;
        alive = false;  // reported to the host; the query gives up
    } else if (next == kEmptyChild) {
        next = stack_pop<ANY>(st, tmax, best, sp, bottom);
        if (next == kEmptyChild) alive = false;
    }
    cur = next;
}

// Test the entries of one leaf (`leaf` a leaf code) against a query; an any-hit query stops
// at its first hit.
template <bool ANY, bool CNT>
__device__ __forceinline__ void leaf_test(const float4* __restrict__ prims, int leaf, const RayPre& r, float tmin,
                                          float tmax, Hit& best, bool& hit_any, TraceWork* work, bool wt) {
    const int first = leaf_first(leaf), cnt = leaf_count(leaf);
    if (CNT) work->prims += cnt;
    if (ANY) {
        for (int e = first; e < first + cnt; e++) {
            if (leaf_entry_any(prims, e, r, tmin, tmax, wt)) {
                hit_any = true;
                break;
            }
        }
    } else {
        for (int e = first; e < first + cnt; e++) leaf_entry(prims, e, r, tmin, tmax, best, wt);
    }
}

// One leaf visit of a live query (`cur` a leaf code): test its entries, then pop the stack.
// An any-hit query ends at its first hit (`hit_any`); every query ends on an empty stack.
template <bool ANY, bool CNT>
__device__ __forceinline__ void leaf_step(const float4* __restrict__ prims, const RayPre& r, float tmin, float tmax,
                                          const LaneStack<ANY>& st, Hit& best, int& cur, int& sp, bool& alive,
                                          bool& hit_any, TraceWork* work, bool wt, int bottom) {
    leaf_test<ANY, CNT>(prims, cur, r, tmin, tmax, best, hit_any, work, wt);
    if (ANY && hit_any) alive = false;
    if (alive) {
        cur = stack_pop<ANY>(st, tmax, best, sp, bottom);
        if (cur == kEmptyChild) alive = false;
    }
}

// One round of the warp-synchronous traversal; every lane of the warp calls it together.
// Phase 1 visits internal nodes until twice as many lanes wait with a leaf as still search for
// one; phase 2 tests the leaves. Waiting for the last searching lane left most of a warp idle on
// incoherent rays (8 of 32 lanes active on the 1.31M-triangle mesh). Frame ms with phase 1
// ending at the last lane / at waiting >= 1x / 2x / 4x / 8x searching: mesh 33.7 / 30.1 / 30.2 / 30.7 / 31.7, slit
// room 86.7 / 82.6 / 81.8 / 81.5 / 82.3, spheres 25.7 / 26.0 / 25.9 / 25.8 / 25.8, Cornell 3.26 / 3.31 / 3.26 / 3.26 /
// 3.28.
// With `spec` (speculative traversal, Aila and Laine 2009), a lane that reaches its first leaf
// parks it in `pend` and keeps descending while some lane of the warp has found no leaf yet, so
// the node phase runs with fuller warps; the parked leaf is tested in phase 2. Closest hits are the minimum of a total order, so the visiting order
// never changes a result; speculation only visits nodes that a tighter bound might have culled.
template <int W, bool ANY, bool CNT>
__device__ __forceinline__ void traverse_round(const float4* __restrict__ nodes, const float4* __restrict__ prims,
                                               bool quant, bool spec, const RayPre& r, float tmin, float tmax,
                                               const LaneStack<ANY>& st, Hit& best, int& cur, int& pend, int& sp,
                                               bool& alive, bool& hit_any, int& overflow, TraceWork* work,
                                               bool wt = false, bool near = false, int bottom = 0) {
    // ---- phase 1: internal nodes, while enough live lanes have found no leaf
    const int live = __popc(__ballot_sync(0xffffffffu, alive));
    for (;;) {
        const int searching = __popc(__ballot_sync(0xffffffffu, alive && cur >= 0 && pend == kEmptyChild));
        if (3 * searching <= live) break;
        if (alive && cur >= 0) {
            node_step<W, ANY, CNT>(nodes, quant, r, tmin, tmax, st, best, cur, sp, alive, overflow, work, near, bottom);
            if (spec) {
                if (!alive && !overflow && pend != kEmptyChild) {
                    alive = true;  // the stack ran empty: only the parked leaf is left
                    cur = pend;
                    pend = kEmptyChild;
                } else if (alive && cur < 0 && pend == kEmptyChild) {
                    pend = cur;  // park the first leaf and keep descending
                    cur = stack_pop<ANY>(st, tmax, best, sp, bottom);
                    if (cur == kEmptyChild) {
                        cur = pend;
                        pend = kEmptyChild;
                    }
                }
            }
        }
    }
    // ---- phase 2: the parked leaf, then the current one (which pops the stack)
    if (alive && pend != kEmptyChild) {
        leaf_test<ANY, CNT>(prims, pend, r, tmin, tmax, best, hit_any, work, wt);
        pend = kEmptyChild;
        if (ANY && hit_any) alive = false;
    }
    if (alive && cur < 0)
        leaf_step<ANY, CNT>(prims, r, tmin, tmax, st, best, cur, sp, alive, hit_any, work, wt, bottom);
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
// Position of the k-th set bit (k from 0, below the mask's count).
__device__ __forceinline__ int nth_bit(unsigned mask, int k) {
    int pos = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const int c = __popc(mask & ((1u << s) - 1u));
        if (k >= c) {
            k -= c;
            pos += s;
            mask >>= s;
        }
    }
    return pos;
}
// The better of two closest hits of one query (the total order of leaf_entry).
__device__ __forceinline__ void merge_hit(Hit& best, const Hit& c) {
    if (c.prim == kMissPrim) return;
    const bool tie = c.prim >= 0 ? (best.prim < 0 || c.prim > best.prim) : (best.prim < 0 && c.prim > best.prim);
    if (best.prim == kMissPrim || c.t < best.t || (c.t == best.t && tie)) best = c;
}
__device__ __forceinline__ float shfl_f(float v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// The end of a persistent traversal: the queue is empty and few lanes of the warp still carry a query.
// Their queries are the long ones (on the meshes a launch ran on for 50 to 200 us after half of its warps
// had ended), so the idle lanes help: each takes the bottom entry of a busy lane's stack, the
// largest subtree left behind, with the ray, and traverses it as its own. A helper's hit is
// merged into its owner's when the helper runs dry (closest hits are the minimum of a total order, so the
// split changes nothing); helpers cull against the owner's hit as of the last round, one ulp
// farther, so that ties still reach the merge. A query ends when its owner and all of its helpers
// have. `has`: the lane carries a query; `end()` finishes the lane's query and returns whether it
// started another (with cur, sp, h, tmin set and alive true).
template <int W, bool ANY, bool CNT, class End>
__device__ __forceinline__ void traverse_tail(const float4* __restrict__ nodes, const float4* __restrict__ prims,
                                              bool quant, RayPre& r, float& tmin, float& tmax,
                                              const LaneStack<ANY>& st, Hit& h, int& cur, int& sp, bool& alive,
                                              bool& occ, int& of, bool has, TraceWork* work, bool wt, bool near,
                                              End&& end) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float full = tmax;       // this lane's own query's bound
    int owner = has ? lane : -1;   // the lane whose query this lane works on
    int bottom = 0, pend = kEmptyChild;
    // a ray that is not finite is not shared: its hits can be NaN, and the last one visited stands
    const bool shares = isfinite(r.ix + r.iy + r.iz + r.ox + r.oy + r.oz);
    while (__any_sync(kAll, owner >= 0)) {
        const unsigned idle = __ballot_sync(kAll, owner < 0);
        const unsigned rich = __ballot_sync(kAll, alive && sp - bottom >= 2 && (shares || owner != lane));
        if (idle != 0 && rich != 0) {
            const int n = min(__popc(idle), __popc(rich));
            const int rank = __popc((owner < 0 ? idle : rich) & lanemask_lt());
            const bool take = owner < 0 && rank < n;
            const bool give = ((rich >> lane) & 1u) && rank < n;
            const int from = take ? nth_bit(rich, rank) : lane;
            int child = kEmptyChild;
            if (give) {
                if constexpr (ANY) child = *st.slot(bottom);
                else child = st.slot(bottom)->x;
                bottom++;
            }
            child = __shfl_sync(kAll, child, from);
            const float bound = ANY || h.prim == kMissPrim ? tmax : __int_as_float(__float_as_int(fmaxf(h.t, 0.f)) + 1);
            const float lim = shfl_f(bound, from), t0 = shfl_f(tmin, from);
            const int of_query = __shfl_sync(kAll, owner, from);
            RayPre v;
            v.o = V{shfl_f(r.o.x, from), shfl_f(r.o.y, from), shfl_f(r.o.z, from)};
            v.d = V{shfl_f(r.d.x, from), shfl_f(r.d.y, from), shfl_f(r.d.z, from)};
            v.ix = shfl_f(r.ix, from); v.iy = shfl_f(r.iy, from); v.iz = shfl_f(r.iz, from);
            v.ox = shfl_f(r.ox, from); v.oy = shfl_f(r.oy, from); v.oz = shfl_f(r.oz, from);
            if (take) {
                r = v;
                tmin = t0;
                tmax = lim;
                owner = of_query;
                h = Hit{lim, 0.f, 0.f, kMissPrim};
                cur = child;
                sp = bottom = 0;
                occ = false;
                of = 0;
                alive = child != kEmptyChild;
            }
        }
        traverse_round<W, ANY, CNT>(nodes, prims, quant, false, r, tmin, tmax, st, h, cur, pend, sp, alive, occ, of,
                                    work, wt, near, bottom);
        // the lanes of one query
        const unsigned group = __match_any_sync(kAll, owner >= 0 ? owner : 32 + lane);
        const unsigned failed = __ballot_sync(kAll, owner >= 0 && of != 0);
        const unsigned hits = __ballot_sync(kAll, ANY && owner >= 0 && occ);
        if ((failed | hits) & group) {  // a query gives up, or is occluded, as a whole
            if (failed & group) of = 1;
            if (hits & group) occ = true;
            alive = false;
        }
        const bool helper = owner >= 0 && owner != lane;
        if constexpr (!ANY) {
            unsigned done = __ballot_sync(kAll, helper && !alive);
            while (done) {
                const int b = __ffs(done) - 1;
                done &= done - 1;
                const Hit c{shfl_f(h.t, b), shfl_f(h.b1, b), shfl_f(h.b2, b), __shfl_sync(kAll, h.prim, b)};
                if (lane == __shfl_sync(kAll, owner, b)) merge_hit(h, c);
            }
            const float bound = h.prim == kMissPrim ? tmax : __int_as_float(__float_as_int(fmaxf(h.t, 0.f)) + 1);
            const float lim = shfl_f(bound, owner >= 0 ? owner : lane);
            if (helper && lim < tmax) {
                tmax = lim;
                if (h.prim != kMissPrim && h.t > lim) h.prim = kMissPrim;
            }
        }
        const unsigned live = __ballot_sync(kAll, alive);
        if (helper && !alive) owner = -1;
        if (owner == lane && !(live & group)) {
            tmax = full;
            bottom = 0;
            if (!end()) owner = -1;
        }
    }
}

// Warp-synchronous traversal: every lane of the warp calls this together (`active` marks the
// lanes that carry a query). Lanes advance through internal nodes in one phase and test
// leaves in the next, re-converging at each phase boundary (the while-while organisation of
// Aila and Laine, HPG 2009), so leaf tests and node visits execute as coherent SIMT
// instructions instead of drifting apart. Closest hit, no refill: the queries that start and end
// together (normals frames, the pick).
template <int W>
__device__ __forceinline__ void traverse(const SceneDevice& sc, const RayPre& r, float tmin, float tmax, bool active,
                                         const LaneStack<false>& st, Hit& best, int& overflow) {
    const bool quant = W >= 4 && sc.node_q != 0, wt = sc.watertight != 0;  // warp-uniform
    best.prim = kMissPrim;
    best.t = tmax;
    int sp = 0;
    int cur = active ? sc.root : kEmptyChild;
    bool alive = active;
    bool hit_any = false;
    int pend = kEmptyChild;
    while (__any_sync(0xffffffffu, alive))
        traverse_round<W, false, false>(sc.nodes, sc.prims, quant, false, r, tmin, tmax, st, best, cur, pend, sp, alive,
                                        hit_any, overflow, nullptr, wt);
}

}  // namespace pt
