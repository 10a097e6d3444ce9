// pt_traverse.cuh -- short-stack closest-hit and any-hit traversal of the
// wide BVH (2, 4 or 8 children per node) on FP32 SIMT cores.
//
// Replaces optixTrace (example/path_tracer/main.cu:80-85,161-166; closest hit,
// tmin 0.001, tmax 1e16) and Emitter::TraceShadowRay (framework/render/
// emitter.h:91-100; terminate on first hit).  Result semantics (shared with
// the CPU oracle): a primitive is hit at tmin < t < tmax; the closest hit is
// the smallest t, ties broken by the smaller primitive id, so the answer does
// not depend on traversal order.  The triangle test is the watertight test of
// Woop, Benthin and Wald (JCGT 2013) evaluated with explicitly rounded
// operations (no FMA contraction), which makes hit ids and distances bit-equal
// to the host restatement.
//
// Memory layout (HBM):
//   node  = 8*K floats: lo_x[K] hi_x[K] lo_y[K] hi_y[K] lo_z[K] hi_z[K]
//           item[K], K unused.  item: a traversal item (below): an inner node's
//           index, a leaf's first slot and count, or kNoItem (empty slot, a
//           point box far away).  Stored swizzled by the node's index
//           (node_swizzle), loaded 16 or 32 bytes at a time (load_node).
//   prim  = 3 float4 per slot: triangle (v0, id) (v1, 0) (v2, 0);
//           sphere (centre, id | 1<<31) (radius, 0, 0, 0) (0);
//           curve piece (c0, id | 1<<31) (r0, r1, u0, kind bits) (c1, u1):
//           a round cone from centre c0 / radius r0 to c1 / r1 covering the
//           curve parameters [u0, u1] of its segment (pt_curve.h).
// Nodes are in breadth-first order, so the first smem_nodes nodes are the
// top levels; those are staged in shared memory once per (persistent) block.
// Width 8 traverses compressed copies of the nodes instead (CwNode below).
#pragma once

#include "pt_curve.h"
#include "pt_device.cuh"

namespace ptd {

constexpr int kShortStack = 16;  // shared-memory entries per thread
constexpr int kSpillStack = kTraversalStackEntries - kShortStack;  // local-memory overflow entries per thread
constexpr float kSlabScale = 1.0000004f;  // 1 + 2*gamma(3): robust slab far bound (Ize 2013)

// Traversal items: a node index (>= 0), a leaf (bit 31 | first << 4 | count)
// or kNoItem.  Leaves must start below 2^27 - 1 (checked at scene upload).
// Nodes hold their children in this form: forming them at every visit (child
// and count) cost the closest hit 105 against 89.5 ms and spilled registers.
constexpr int kNoItem = -1;
PT_DI int make_leaf(int first, int count) { return (int)(0x80000000u | ((uint32_t)first << 4) | (uint32_t)count); }
PT_DI bool is_leaf(int item) { return item < 0 && item != kNoItem; }
PT_DI int leaf_first(int item) { return (int)(((uint32_t)item >> 4) & 0x7ffffffu); }
PT_DI int leaf_count(int item) { return item & 15; }

struct TraceResult {
    float t;
    int prim;
    float u, v;
};

struct RayWT {  // per-ray constants of the watertight test
    int kx, ky, kz;
    float sx, sy, sz;
};

PT_DI float sel3(float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

PT_DI RayWT ray_wt(float3 d) {
    RayWT r;
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    r.kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    r.kx = r.kz + 1 == 3 ? 0 : r.kz + 1;
    r.ky = r.kx + 1 == 3 ? 0 : r.kx + 1;
    float dz = sel3(d, r.kz);
    if (dz < 0.f) {
        int t = r.kx;
        r.kx = r.ky;
        r.ky = t;
    }
    r.sx = __fdiv_rn(sel3(d, r.kx), dz);
    r.sy = __fdiv_rn(sel3(d, r.ky), dz);
    r.sz = __frcp_rn(dz);
    return r;
}

// Watertight ray/triangle test with explicitly rounded operations.
PT_DI bool intersect_triangle(float3 o, const RayWT &w, float3 p0, float3 p1, float3 p2, float tmin, float tmax,
                              float &t_out, float &u_out, float &v_out) {
    float3 A = f3(__fsub_rn(p0.x, o.x), __fsub_rn(p0.y, o.y), __fsub_rn(p0.z, o.z));
    float3 B = f3(__fsub_rn(p1.x, o.x), __fsub_rn(p1.y, o.y), __fsub_rn(p1.z, o.z));
    float3 C = f3(__fsub_rn(p2.x, o.x), __fsub_rn(p2.y, o.y), __fsub_rn(p2.z, o.z));
    float Akz = sel3(A, w.kz), Bkz = sel3(B, w.kz), Ckz = sel3(C, w.kz);
    float Ax = __fsub_rn(sel3(A, w.kx), __fmul_rn(w.sx, Akz));
    float Ay = __fsub_rn(sel3(A, w.ky), __fmul_rn(w.sy, Akz));
    float Bx = __fsub_rn(sel3(B, w.kx), __fmul_rn(w.sx, Bkz));
    float By = __fsub_rn(sel3(B, w.ky), __fmul_rn(w.sy, Bkz));
    float Cx = __fsub_rn(sel3(C, w.kx), __fmul_rn(w.sx, Ckz));
    float Cy = __fsub_rn(sel3(C, w.ky), __fmul_rn(w.sy, Ckz));
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (U == 0.f || V == 0.f || W == 0.f) {  // double-precision fallback on edges
        U = __double2float_rn(__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx)));
        V = __double2float_rn(__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx)));
        W = __double2float_rn(__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax)));
    }
    if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
    float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.f) return false;
    float Az = __fmul_rn(w.sz, Akz), Bz = __fmul_rn(w.sz, Bkz), Cz = __fmul_rn(w.sz, Ckz);
    float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    float rcp = __frcp_rn(det);
    float t = __fmul_rn(T, rcp);
    if (!(t > tmin && t < tmax)) return false;
    t_out = t;
    u_out = __fmul_rn(V, rcp);
    v_out = __fmul_rn(W, rcp);
    return true;
}

// Ray/sphere with the two precision improvements of Haines, Guenther and
// Akenine-Moeller ("Precision Improvements for Ray/Sphere Intersection", Ray
// Tracing Gems, 2019): the discriminant from the distance of the closest
// approach to the centre, r^2 - |f + (b'/a) d|^2, instead of b^2 - ac (which
// cancels for distant or small spheres), and the two roots as c/q and q/a with
// q = b' + sign(b') sqrt(a * disc) (no subtraction of nearly equal values).
// The roots are then accurate to a few ulp of t, so a hit always lies inside
// the sphere's (padded) bounding box and the result cannot depend on which
// BVH nodes the traversal culls.  Every step is rounded separately, as in
// the oracle's host build of the same formula.
PT_DI bool intersect_sphere(float3 o, float3 d, float3 c, float r, float tmin, float tmax, float &t_out) {
    const float3 f = f3(__fsub_rn(o.x, c.x), __fsub_rn(o.y, c.y), __fsub_rn(o.z, c.z));
    const float a = __fadd_rn(__fadd_rn(__fmul_rn(d.x, d.x), __fmul_rn(d.y, d.y)), __fmul_rn(d.z, d.z));
    const float bp = -__fadd_rn(__fadd_rn(__fmul_rn(f.x, d.x), __fmul_rn(f.y, d.y)), __fmul_rn(f.z, d.z));
    const float s = __fdiv_rn(bp, a);
    const float3 l = f3(__fadd_rn(f.x, __fmul_rn(s, d.x)), __fadd_rn(f.y, __fmul_rn(s, d.y)),
                        __fadd_rn(f.z, __fmul_rn(s, d.z)));
    const float rr = __fmul_rn(r, r);
    const float disc = __fsub_rn(rr, __fadd_rn(__fadd_rn(__fmul_rn(l.x, l.x), __fmul_rn(l.y, l.y)), __fmul_rn(l.z, l.z)));
    if (!(disc >= 0.f)) return false;
    const float cc = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(f.x, f.x), __fmul_rn(f.y, f.y)), __fmul_rn(f.z, f.z)), rr);
    const float q = __fadd_rn(bp, copysignf(__fsqrt_rn(__fmul_rn(a, disc)), bp));
    float t0 = __fdiv_rn(cc, q), t1 = __fdiv_rn(q, a);
    if (t0 > t1) {
        const float tt = t0;
        t0 = t1;
        t1 = tt;
    }
    if (t0 > tmin && t0 < tmax) {
        t_out = t0;
        return true;
    }
    if (t1 > tmin && t1 < tmax) {
        t_out = t1;
        return true;
    }
    return false;
}

// ---------------------------------------------------------------- curve pieces
PT_DI float dot_rn(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
PT_DI float3 sub_rn(float3 a, float3 b) { return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
PT_DI float3 madd_rn(float3 a, float s, float3 b) {  // a + s*b, rounded per step
    return f3(__fadd_rn(a.x, __fmul_rn(s, b.x)), __fadd_rn(a.y, __fmul_rn(s, b.y)), __fadd_rn(a.z, __fmul_rn(s, b.z)));
}

// Entry into a sphere, the ray origin first moved to the point of closest
// approach (Haines et al., "Precision Improvements for Ray/Sphere
// Intersection", Ray Tracing Gems 2019), which keeps hair-thin spheres exact
// for distant origins.  Only the entering root counts.
PT_DI bool curve_sphere_entry(float3 o, float3 d, float dd, float3 c, float r, float tmin, float tmax, float &t_out) {
    const float3 f = sub_rn(o, c);
    const float tc = __fdiv_rn(-dot_rn(f, d), dd);
    const float3 l = madd_rn(f, tc, d);
    const float h = __fsub_rn(__fmul_rn(r, r), dot_rn(l, l));
    if (!(h >= 0.f)) return false;
    const float t = __fsub_rn(tc, __fsqrt_rn(__fdiv_rn(h, dd)));
    if (!(t > tmin && t < tmax)) return false;
    t_out = t;
    return true;
}

// Round-cone piece: the lateral surface of the cone frustum between the
// planes through c0 and c1 normal to the axis (radius linear along the
// axis), plus spheres at the ends that the kind bits ask for.  The frustum
// quadratic is formed from the components normal to the axis, origin moved to
// the closest approach to c0; its entering root is (-B - sqrt(B^2 - AC)) / A
// whatever the sign of A.  Returns the smallest entering t in (tmin, tmax)
// and the curve parameter there (projection onto the axis, mapped to [u0, u1]).
PT_DI bool intersect_curve_piece(float3 o, float3 d, float4 a, float4 b, float4 c, float tmin, float tmax, float &t_out,
                                 float &u_out) {
    const int kind = __float_as_int(b.w);
    const float3 c0 = xyz(a), c1 = xyz(c);
    const float r0 = b.x, r1 = b.y, u0 = b.z, u1 = c.w;
    const float dd = dot_rn(d, d);
    bool hit = false;
    float best = tmax, bu = 0.f, t;
    if ((kind & kPieceSphere0) && curve_sphere_entry(o, d, dd, c0, r0, tmin, best, t)) {
        hit = true;
        best = t;
        bu = u0;
    }
    if ((kind & kPieceSphere1) && curve_sphere_entry(o, d, dd, c1, r1, tmin, best, t)) {
        hit = true;
        best = t;
        bu = u1;
    }
    const float3 e = sub_rn(c1, c0);
    const float len = __fsqrt_rn(dot_rn(e, e));
    if (len > 0.f) {
        const float inv_len = __frcp_rn(len);
        const float3 ax = f3(__fmul_rn(e.x, inv_len), __fmul_rn(e.y, inv_len), __fmul_rn(e.z, inv_len));
        const float k = __fmul_rn(__fsub_rn(r1, r0), inv_len);  // dr / dz
        const float3 f = sub_rn(o, c0);
        const float tc = __fdiv_rn(-dot_rn(f, d), dd);
        const float3 w = madd_rn(f, tc, d);
        const float we = dot_rn(w, ax), de = dot_rn(d, ax);
        const float3 wp = madd_rn(w, -we, ax), dp = madd_rn(d, -de, ax);
        const float rz = __fadd_rn(r0, __fmul_rn(k, we));
        const float kde = __fmul_rn(k, de);
        const float A = __fsub_rn(dot_rn(dp, dp), __fmul_rn(kde, kde));
        const float B = __fsub_rn(dot_rn(wp, dp), __fmul_rn(kde, rz));
        const float C = __fsub_rn(dot_rn(wp, wp), __fmul_rn(rz, rz));
        const float disc = __fsub_rn(__fmul_rn(B, B), __fmul_rn(A, C));
        if (disc >= 0.f && A != 0.f) {
            const float tp = __fdiv_rn(__fsub_rn(-B, __fsqrt_rn(disc)), A);
            const float z = __fadd_rn(we, __fmul_rn(tp, de));
            const float tt = __fadd_rn(tc, tp);
            if (z >= 0.f && z <= len && tt > tmin && tt < best) {
                hit = true;
                best = tt;
                bu = __fadd_rn(u0, __fmul_rn(__fmul_rn(z, inv_len), __fsub_rn(u1, u0)));
            }
        }
    }
    if (!hit) return false;
    if (kind & kPieceClampU) bu = fminf(fmaxf(bu, kCurveUMin), kCurveUMax);
    t_out = best;
    u_out = bu;
    return true;
}

PT_DI float3 safe_inv(float3 d) {
    return f3(d.x != 0.f ? __frcp_rn(d.x) : copysignf(1e30f, d.x), d.y != 0.f ? __frcp_rn(d.y) : copysignf(1e30f, d.y),
              d.z != 0.f ? __frcp_rn(d.z) : copysignf(1e30f, d.z));
}

// Word w of node i is stored at word w ^ node_swizzle<K>(i) of its record.  The
// lanes of a warp read the same words of different nodes at a time; unswizzled
// these lie in the same banks of L1, one lane per cycle.  112-byte gathers of a
// 128-byte node by 16 lanes of a warp: 1.82 ms unswizzled, 0.97 swizzled while the
// nodes are in L1; 2.21 and 1.82 when they come from L2.  The 1M-triangle field at
// 1080p, 64 spp: closest / any hit 86.8 / 25.2 ms, so 80.0 / 22.1.  Width 4 moves
// 16-byte pieces, width 2 32-byte halves; 8-wide nodes are read as 96-byte copies,
// which fall on different banks by themselves.
template <int K>
PT_HDI constexpr uint32_t node_swizzle(uint32_t i) {
    return K == 4 ? (i & 7) << 2 : K == 2 ? (i & 2) << 2 : 0;
}

// A node as a ray sees it.  Widths 2 and 8: low and high planes, then items.
// Width 4: near and far planes by the ray's octant.
template <int K>
struct WideNode {
    float f[8 * K];
    PT_DI float p0(int axis, int c) const { return f[2 * axis * K + c]; }
    PT_DI float p1(int axis, int c) const { return f[(2 * axis + 1) * K + c]; }
    PT_DI int item(int c) const { return __float_as_int(f[6 * K + c]); }
};

// BVH nodes and primitive records are read many times per wave while the ray
// state streams through once: node and primitive loads ask L1 to evict them
// last, the ray state's loads and stores ask for evict-first (ld/st .cs).
// Measured on the 1M-triangle scene: closest hit 1.1 % faster than plain
// loads; an additional L2 evict-last access policy on the BVH loads gave
// back half of that.
PT_DI float4 ld_bvh(const float4 *p) {
    float4 v;
    asm("ld.global.nc.L1::evict_last.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p));
    return v;
}
// 32 bytes per load (256-bit global loads, sm_100 and later): a node is
// 32 * K bytes at a 32-byte-aligned offset of a cudaMalloc'd array.
PT_DI void ld_bvh8(const float4 *p, float *f) {
    asm("ld.global.nc.L1::evict_last.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
        : "l"(p));
}

// 32 bytes of ray state, streaming (evict-first), and the same store.
PT_DI void ld_stream8(const float4 *p, float4 &a, float4 &b) {
    asm volatile("ld.global.L1::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
PT_DI void ld8(const float4 *p, float4 &a, float4 &b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
PT_DI void st8(float4 *p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

template <typename T>
PT_DI T ld_stream(const T *p) {
    return __ldcs(p);
}
template <typename T>
PT_DI void st_stream(T *p, T v) {
    __stcs(p, v);
}

// The 7*K floats in use, from global (GLOBAL) or shared memory.  Width 4 loads 16
// bytes at a time and picks each axis's near and far planes by address, which
// takes 24 minima and maxima out of the slab test: 1.5 to 3 % of the small frames'
// time against 32-byte loads and min / max (which ask less of L1: equal at 64 spp).
template <int K, bool GLOBAL>
PT_DI void load_node(const float4 *__restrict__ nodes, int item, int oct, WideNode<K> &n) {
    const uint32_t swz = 4 * node_swizzle<K>(item);  // in bytes; the array in global memory is aligned to a record
    const float4 *rec = nodes + (size_t)item * 2 * K;
    const uintptr_t p = reinterpret_cast<uintptr_t>(rec) | swz;
    const auto load4 = [&](int i, uint32_t at) {
        const float4 v = GLOBAL ? ld_bvh(reinterpret_cast<const float4 *>(p ^ at)) : rec[(at ^ swz) / 16];
        n.f[4 * i + 0] = v.x;
        n.f[4 * i + 1] = v.y;
        n.f[4 * i + 2] = v.z;
        n.f[4 * i + 3] = v.w;
    };
    if constexpr (K == 4) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const uint32_t side = (oct << (4 - a)) & 16;
            load4(2 * a, (32 * a) | side);
            load4(2 * a + 1, ((32 * a) | side) ^ 16);
        }
        load4(6, 96);
    } else if constexpr (GLOBAL) {
        static_assert(K == 2, "8-wide nodes are read compressed");
        ld_bvh8(reinterpret_cast<const float4 *>(p), n.f);
        load4(2, 32);
        load4(3, 48);
    } else {
#pragma unroll
        for (int i = 0; i < 2 * K; i++) load4(i, 16 * i);
    }
}

// Compressed 8-wide nodes: 96 bytes (6 float4) per node, after the quantised
// wide nodes of Ylitie, Karras and Laine ("Efficient Incoherent Ray Traversal
// on GPUs Through Compressed Wide BVHs", HPG 2017), with 32-bit child items:
//   q0      xyz: grid origin p; w bits: biased exponents of the per-axis cell
//           sizes 2^e (bytes 0-2), mask of the occupied slots (byte 3)
//   q1..q3  axis x, y, z: low cells of slots 0-7 (8 bytes), high cells (8 bytes)
//   q4, q5  child items of slots 0-7 (inner node index, leaf item or kNoItem)
// Slot c's box is [fma(lo, 2^e, p), fma(hi, 2^e, p)] per axis; the builder
// picks the cells so that these bounds enclose the child's padded float box.
// Slot s holds the child that rays of direction octant s (bit 0: d.x < 0,
// bit 1: d.y < 0, bit 2: d.z < 0) should visit first, and a ray takes the hit
// children in the order slot ^ octant: no sorting of the children.
constexpr int kCwFloat4 = 6;

// Cell `c` (0-7) of the 8 bytes held by the words (w0, w1): the byte is
// placed in the mantissa of 2^23 with one byte permute, and 2^23 is taken
// off again (exact), which avoids the slower integer-to-float conversion.
PT_DI float cw_cell(uint32_t w0, uint32_t w1, int c) {
    const uint32_t v = __byte_perm(c & 4 ? w1 : w0, 0x4b000000u, 0x7650u | static_cast<uint32_t>(c & 3));
    return __fsub_rn(__uint_as_float(v), 8388608.f);
}
PT_DI int cw_pick(int4 i0, int4 i1, int c) {
    const int4 h = c & 4 ? i1 : i0;
    return c & 2 ? (c & 1 ? h.w : h.z) : (c & 1 ? h.y : h.x);
}

// Slab test of the 8 children of compressed node `p`, in visiting order:
// entry k is slot k ^ oct.  ci[k] = child item (kNoItem: missed or empty),
// ct[k] = entry distance.  fast: origin within the magnitude the boxes were
// padded for, so t = fma(cell, 2^e * inv, (p - o) * inv) is conservative
// (its error, at most about 2 ulp of |p - o|, stays inside the padding);
// otherwise each bound is formed as in the build and tested as a float box.
PT_DI void cw_children(const float4 *p, float3 o, float3 inv, bool fast, float tmin, float tlimit, int oct, int *ci,
                       float *ct) {
    float f[24];  // 96 bytes at a 32-byte-aligned offset: three 256-bit loads
    ld_bvh8(p, f);
    ld_bvh8(p + 2, f + 8);
    ld_bvh8(p + 4, f + 16);
    const float4 q0 = make_float4(f[0], f[1], f[2], f[3]), q1 = make_float4(f[4], f[5], f[6], f[7]),
                 q2 = make_float4(f[8], f[9], f[10], f[11]), q3 = make_float4(f[12], f[13], f[14], f[15]);
    const int4 i0 = make_int4(__float_as_int(f[16]), __float_as_int(f[17]), __float_as_int(f[18]), __float_as_int(f[19])),
               i1 = make_int4(__float_as_int(f[20]), __float_as_int(f[21]), __float_as_int(f[22]), __float_as_int(f[23]));
    const uint32_t meta = __float_as_uint(q0.w);
    const float sx = __uint_as_float((meta & 0xffu) << 23), sy = __uint_as_float(((meta >> 8) & 0xffu) << 23),
                sz = __uint_as_float(((meta >> 16) & 0xffu) << 23);
    const uint32_t occupied = meta >> 24;
    const float ax = __fmul_rn(sx, inv.x), ay = __fmul_rn(sy, inv.y), az = __fmul_rn(sz, inv.z);
    const float bx = __fmul_rn(__fsub_rn(q0.x, o.x), inv.x), by = __fmul_rn(__fsub_rn(q0.y, o.y), inv.y),
                bz = __fmul_rn(__fsub_rn(q0.z, o.z), inv.z);
    const uint32_t lx0 = __float_as_uint(q1.x), lx1 = __float_as_uint(q1.y), hx0 = __float_as_uint(q1.z),
                   hx1 = __float_as_uint(q1.w);
    const uint32_t ly0 = __float_as_uint(q2.x), ly1 = __float_as_uint(q2.y), hy0 = __float_as_uint(q2.z),
                   hy1 = __float_as_uint(q2.w);
    const uint32_t lz0 = __float_as_uint(q3.x), lz1 = __float_as_uint(q3.y), hz0 = __float_as_uint(q3.z),
                   hz1 = __float_as_uint(q3.w);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int c = k ^ oct;
        ci[k] = kNoItem;
        ct[k] = __int_as_float(0x7f800000);
        if (!((occupied >> c) & 1u)) continue;
        const float clx = cw_cell(lx0, lx1, c), chx = cw_cell(hx0, hx1, c);
        const float cly = cw_cell(ly0, ly1, c), chy = cw_cell(hy0, hy1, c);
        const float clz = cw_cell(lz0, lz1, c), chz = cw_cell(hz0, hz1, c);
        float tx0, tx1, ty0, ty1, tz0, tz1;
        if (fast) {
            tx0 = __fmaf_rn(clx, ax, bx);
            tx1 = __fmaf_rn(chx, ax, bx);
            ty0 = __fmaf_rn(cly, ay, by);
            ty1 = __fmaf_rn(chy, ay, by);
            tz0 = __fmaf_rn(clz, az, bz);
            tz1 = __fmaf_rn(chz, az, bz);
        } else {
            tx0 = __fmul_rn(__fsub_rn(__fmaf_rn(clx, sx, q0.x), o.x), inv.x);
            tx1 = __fmul_rn(__fsub_rn(__fmaf_rn(chx, sx, q0.x), o.x), inv.x);
            ty0 = __fmul_rn(__fsub_rn(__fmaf_rn(cly, sy, q0.y), o.y), inv.y);
            ty1 = __fmul_rn(__fsub_rn(__fmaf_rn(chy, sy, q0.y), o.y), inv.y);
            tz0 = __fmul_rn(__fsub_rn(__fmaf_rn(clz, sz, q0.z), o.z), inv.z);
            tz1 = __fmul_rn(__fsub_rn(__fmaf_rn(chz, sz, q0.z), o.z), inv.z);
        }
        const float tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), tmin));
        float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
        tf = fminf(__fmul_rn(tf, kSlabScale), tlimit);
        if (!(tn <= tf)) continue;
        ci[k] = cw_pick(i0, i1, c);
        ct[k] = tn;
    }
}

// Per-thread traversal stack: kShortStack entries in shared memory (strided by
// the block size to avoid bank conflicts), the rest in local memory.  Closest
// hit keeps (item, entry distance) and drops entries beyond its hit when they
// are popped; any hit, whose limit never moves, keeps the item alone (any hit
// 25.8 -> 25.3 ms a 64-spp 1080p frame of the 1M-triangle field).  Closest /
// any hit ms with 8, 10, 12, 16, 20, 24 entries in shared memory: 90.3 / 26.4,
// 87.5 / 25.6, 86.3 / 25.2, 86.0 / 25.3, 86.7 / 25.3, 88.3 / 25.3 (what the
// stack takes, L1 loses).
template <bool ANY>
struct StackEntry {
    using type = int2;
    PT_DI static int2 make(int item, float t) { return make_int2(item, __float_as_int(t)); }
    PT_DI static int item(int2 e) { return e.x; }
    PT_DI static bool within(int2 e, float limit) { return __int_as_float(e.y) <= limit; }
};
template <>
struct StackEntry<true> {
    using type = int;
    PT_DI static int make(int item, float) { return item; }
    PT_DI static int item(int e) { return e; }
    PT_DI static bool within(int, float) { return true; }
};
template <bool ANY>
struct ShortStack {
    using E = StackEntry<ANY>;
    typename E::type *smem;  // base + threadIdx.x
    int stride;
    typename E::type spill[kSpillStack];
    int sp;
    PT_DI void push(int item, float t, uint32_t &overflow) {
        if (sp < kShortStack) smem[sp * stride] = E::make(item, t);
        else if (sp < kShortStack + kSpillStack) spill[sp - kShortStack] = E::make(item, t);
        else {  // cannot happen for trees of depth <= 32 (width 4), 13 (width 8); reported, entry dropped
            overflow = 1;
            return;
        }
        sp++;
    }
    // room for n entries without a check for each: push_short may be used
    PT_DI bool short_room(int n) const { return sp + n <= kShortStack; }
    PT_DI void push_short(int item, float t) {
        smem[sp * stride] = E::make(item, t);
        sp++;
    }
    // the topmost entry no farther than `limit`, or kNoItem
    PT_DI int pop(float limit) {
        while (sp > 0) {
            sp--;
            const typename E::type e = sp < kShortStack ? smem[sp * stride] : spill[sp - kShortStack];
            if (E::within(e, limit)) return E::item(e);
        }
        return kNoItem;
    }
};
constexpr int stack_entry_bytes(bool any) { return any ? 4 : 8; }

// Lanes refill their ray when at most this many lanes of the warp are busy.
constexpr int kRefillBusyMax = 20;
// The node phase ends when at most this many lanes still step towards their
// first leaf (and some lane holds one): the warp does not run on for its
// slowest lanes.  1M-triangle field, 1080p, 64 spp, closest / any hit ms:
// waiting for all lanes 119.8 / 35.4; 2 lanes left 111.7 / 32.6, 4 109.2 / 31.6,
// 8 107.8 / 30.9, 12 109.1 / 30.9, 16 112.8 / 31.8.
constexpr int kNodeWaitMax = 8;

// Persistent "while-while" traversal (after Aila & Laine, HPG 2009), adapted
// to wide nodes with inline leaves.  Each warp keeps 32 rays in flight:
//   refill   when at most kRefillBusyMax lanes are busy, the idle lanes take
//            new rays with one atomic per warp;
//   nodes    lanes step through inner nodes until all but a few busy lanes have
//            found a leaf (it is postponed) or run out of work;
//   leaves   lanes intersect their postponed leaf (any hit: also the leaves
//            that follow it on the stack, since a hit ends the ray; closest hit
//            returns to the nodes after one: 105.6 against 107.8 ms);
//   finish   lanes without work store their result and become idle.
// Children are slab-tested (robust far bound), sorted by entry distance; the
// nearest is the next item, the others go on the stack with their distance,
// which is re-checked against the current closest hit when popped.
//
// Src provides: count(), load(i, o, d, tmin, tmax, tag), root(tag) (the node
// the ray starts at), store(i, tag, result).  A load that leaves tmin and tmax
// alone (extension rays: always 0.001 and 1e16) keeps them out of registers.
// FORM: without kCurves the leaf test has no curve-piece branch (a record with
// non-zero kind bits is then treated as a sphere), so that scenes without curves
// run the smaller kernel; without kStaged every node comes from global memory (the
// test for a staged one costs 1 to 5 %: 1M rays 772 -> 737 us).
enum TraceForm : int { kCurves = 1, kStaged = 2 };
template <int K, bool ANY, bool COUNT, class Src, int FORM = 0>
PT_DI void trace_persistent(const DevScene &s, const float4 *snodes, void *sstack_base, Src &src, uint32_t *work,
                            uint32_t *ovf_flag, unsigned long long *stat_nodes, unsigned long long *stat_prims,
                            unsigned long long *stat_rays) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t n = src.count();
    ShortStack<ANY> st;
    st.smem = static_cast<typename StackEntry<ANY>::type *>(sstack_base) + threadIdx.x;
    st.stride = blockDim.x;
    st.sp = 0;
    bool active = false, exhausted = false;
    uint32_t idx = 0, tag = 0;
    float3 o = f3s(0.f), d = f3s(0.f), inv = f3s(0.f), oi = f3s(0.f);
    bool fma_slab = false;
    int oct = 0;  // direction octant: signs of inv
    RayWT w{0, 1, 2, 0.f, 0.f, 1.f};
    float tmin = 0.001f, tmax = 1e16f;  // the extension rays' range (main.cu:80-85)
    TraceResult best{0.f, -1, 0.f, 0.f};
    int item = kNoItem, leaf = kNoItem;
    uint32_t nodes = 0, prims = 0, rays = 0, ovf = 0;

    auto pop_valid = [&]() -> int { return st.pop(best.t * kSlabScale); };

    for (;;) {
        unsigned busy = __ballot_sync(FULL, active);
        if (!exhausted && __popc(busy) <= kRefillBusyMax) {
            unsigned idle = ~busy;
            uint32_t cnt = __popc(idle);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, cnt);
            base = __shfl_sync(FULL, base, 0);
            if (!active) {
                uint32_t r = base + __popc(idle & lt);
                if (r < n) {
                    idx = r;
                    src.load(r, o, d, tmin, tmax, tag);
                    w = ray_wt(d);
                    inv = safe_inv(d);
                    oi = f3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
                    // the FMA slab form is conservative for origins inside the
                    // magnitude the boxes were padded for
                    fma_slab = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z)) <= s.pad_mag;
                    oct = (__float_as_uint(inv.x) >> 31) | (__float_as_uint(inv.y) >> 31) << 1 |
                          (__float_as_uint(inv.z) >> 31) << 2;
                    best.t = tmax;
                    best.prim = -1;
                    best.u = best.v = 0.f;
                    item = src.root(tag);
                    leaf = kNoItem;
                    st.sp = 0;
                    active = true;
                    if (COUNT) rays++;
                }
            }
            if (base + cnt >= n) exhausted = true;
            busy = __ballot_sync(FULL, active);
        }
        if (busy == 0) break;

        // Inner nodes.  A lane keeps stepping while its current item is an
        // inner node, even after it has postponed a leaf (speculative
        // traversal); a lane that waits for its first leaf can always step.
        for (;;) {
            const bool can_step = active && item >= 0;
            const unsigned wait = __ballot_sync(FULL, can_step && leaf == kNoItem);
            if (wait == 0 || (__popc(wait) <= kNodeWaitMax && __any_sync(FULL, leaf != kNoItem))) break;
            if (!can_step) continue;
            if constexpr (K == 8) {  // compressed node: children come in the octant's visiting order
                if (COUNT) nodes++;
                int ci[8];
                float ct[8];
                cw_children(s.cnodes + (size_t)item * kCwFloat4, o, inv, fma_slab, tmin, best.t * kSlabScale, oct, ci,
                            ct);
                // the first hit child is descended, the later ones pushed (popped in visiting order)
                int next = kNoItem;
                float next_t = 0.f;
                const bool room = st.short_room(7);
#pragma unroll
                for (int i = 7; i >= 0; i--) {
                    if (ci[i] == kNoItem) continue;
                    if (next != kNoItem) {
                        if (room) st.push_short(next, next_t);
                        else st.push(next, next_t, ovf);
                    }
                    next = ci[i];
                    next_t = ct[i];
                }
                item = next != kNoItem ? next : pop_valid();
            } else {
                WideNode<K> nd;
                if ((FORM & kStaged) != 0 && item < static_cast<int>(s.smem_nodes)) load_node<K, false>(snodes, item, oct, nd);
                else load_node<K, true>(s.nodes, item, oct, nd);
                if (COUNT) nodes++;
                int ci[K];
                float ct[K];
                const float tlimit = best.t * kSlabScale;
#pragma unroll
                for (int c = 0; c < K; c++) {
                    ci[c] = kNoItem;
                    ct[c] = __int_as_float(0x7f800000);
                    float tx0, tx1, ty0, ty1, tz0, tz1;
                    if (fma_slab) {  // t = lo * inv - o * inv: one rounding, conservative within pad_mag
                        tx0 = __fmaf_rn(nd.p0(0, c), inv.x, -oi.x);
                        tx1 = __fmaf_rn(nd.p1(0, c), inv.x, -oi.x);
                        ty0 = __fmaf_rn(nd.p0(1, c), inv.y, -oi.y);
                        ty1 = __fmaf_rn(nd.p1(1, c), inv.y, -oi.y);
                        tz0 = __fmaf_rn(nd.p0(2, c), inv.z, -oi.z);
                        tz1 = __fmaf_rn(nd.p1(2, c), inv.z, -oi.z);
                    } else {
                        tx0 = (nd.p0(0, c) - o.x) * inv.x;
                        tx1 = (nd.p1(0, c) - o.x) * inv.x;
                        ty0 = (nd.p0(1, c) - o.y) * inv.y;
                        ty1 = (nd.p1(1, c) - o.y) * inv.y;
                        tz0 = (nd.p0(2, c) - o.z) * inv.z;
                        tz1 = (nd.p1(2, c) - o.z) * inv.z;
                    }
                    const auto lower = [](float a, float b) { return K == 4 ? a : fminf(a, b); };
                    const auto upper = [](float a, float b) { return K == 4 ? b : fmaxf(a, b); };
                    float tn = fmaxf(fmaxf(lower(tx0, tx1), lower(ty0, ty1)), fmaxf(lower(tz0, tz1), tmin));
                    float tf = fminf(fminf(upper(tx0, tx1), upper(ty0, ty1)), upper(tz0, tz1));
                    tf = fminf(tf * kSlabScale, tlimit);
                    if (!(tn <= tf)) continue;
                    ci[c] = nd.item(c);  // an empty slot's stays kNoItem whatever its box says
                    ct[c] = tn;
                }
                // closest hit: nearest child first (sorting network); any hit: order
                // does not matter, the children are taken as they come
#pragma unroll
                for (int i = 1; i < (ANY ? 1 : K); i++) {
#pragma unroll
                    for (int j = i; j > 0; j--) {
                        if (ct[j] < ct[j - 1]) {
                            float tt = ct[j];
                            ct[j] = ct[j - 1];
                            ct[j - 1] = tt;
                            int ti = ci[j];
                            ci[j] = ci[j - 1];
                            ci[j - 1] = ti;
                        }
                    }
                }
                if (ANY) {  // unsorted: the first hit child is descended, the others pushed
#pragma unroll
                    for (int i = 1; i < K; i++)
                        if (ci[0] == kNoItem && ci[i] != kNoItem) {
                            ci[0] = ci[i];
                            ci[i] = kNoItem;
                        }
                }
                // one check for the whole node while the short stack has room
                // (a check per push: closest / any hit 89.5 / 27.8 ms, so 85.9 / 25.8)
                if (st.short_room(K - 1)) {
#pragma unroll
                    for (int i = K - 1; i >= 1; i--)
                        if (ci[i] != kNoItem) st.push_short(ci[i], ct[i]);
                } else {
#pragma unroll
                    for (int i = K - 1; i >= 1; i--)
                        if (ci[i] != kNoItem) st.push(ci[i], ct[i], ovf);
                }
                item = ci[0] != kNoItem ? ci[0] : pop_valid();
            }
            if (is_leaf(item) && leaf == kNoItem) {  // postpone the first leaf
                leaf = item;
                item = pop_valid();
            }
        }

        // leaves
        if (active) {
            while (leaf != kNoItem) {
                const int first = leaf_first(leaf), cnt = leaf_count(leaf);
                for (int j = 0; j < cnt; j++) {
                    const float4 *pr = s.prims + (size_t)(first + j) * 3;
                    float4 a = ld_bvh(pr);
                    float4 b = ld_bvh(pr + 1);
                    if (COUNT) prims++;
                    int pid = __float_as_int(a.w);
                    float t, u = 0.f, v = 0.f;
                    float tlim = best.prim < 0 ? tmax : __int_as_float(__float_as_int(best.t) + 1);
                    bool hit;
                    if (pid >= 0) {
                        float4 cc = ld_bvh(pr + 2);
                        hit = intersect_triangle(o, w, xyz(a), xyz(b), xyz(cc), tmin, tlim, t, u, v);
                    } else if ((FORM & kCurves) == 0 || __float_as_int(b.w) == 0) {
                        pid &= 0x7fffffff;
                        hit = intersect_sphere(o, d, xyz(a), b.x, tmin, tlim, t);
                    } else {
                        pid &= 0x7fffffff;
                        float4 cc = ld_bvh(pr + 2);
                        hit = intersect_curve_piece(o, d, a, b, cc, tmin, tlim, t, u);
                    }
                    if (!hit) continue;
                    if (ANY) {
                        best.t = t;
                        best.prim = pid;
                        break;
                    }
                    if (t < best.t || pid < best.prim) {
                        best.t = t;
                        best.prim = pid;
                        best.u = u;
                        best.v = v;
                    }
                }
                leaf = kNoItem;
                if (ANY && best.prim >= 0) {  // any hit ends the ray
                    item = kNoItem;
                    st.sp = 0;
                    break;
                }
                if (is_leaf(item)) {
                    leaf = item;
                    item = pop_valid();
                }
                if (!ANY) break;
            }
            if (item == kNoItem && leaf == kNoItem) {
                src.store(idx, tag, best);
                active = false;
            }
        }
    }
    if (ovf) atomicOr(ovf_flag, 1u);
    if (COUNT) {
        for (int off = 16; off > 0; off >>= 1) {
            nodes += __shfl_xor_sync(FULL, nodes, off);
            prims += __shfl_xor_sync(FULL, prims, off);
            rays += __shfl_xor_sync(FULL, rays, off);
        }
        if (lane == 0) {
            atomicAdd(stat_nodes, (unsigned long long)nodes);
            atomicAdd(stat_prims, (unsigned long long)prims);
            atomicAdd(stat_rays, (unsigned long long)rays);
        }
    }
}

}  // namespace ptd
