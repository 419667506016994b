// pbg_walk.cuh -- one ray's walk through a two-wide BVH (shared by the
// ray-bvh kernels and the batched many-scene pipeline).
//
// Private stack, nearest child first, leaf children tested as soon as their
// box is hit.  Box test: slab form with t = (bound - o) / d and the far
// distance widened by 1 + 2*gamma(3), conservative for the (already padded)
// boxes.  Degenerate triangles sit in front of the leaf records and are
// tested by every ray.
#pragma once
#include "pbg_count.cuh"
#include "pbg_exact.cuh"
#include "pbg_internal.h"

namespace pbg {

#ifdef __CUDACC__

constexpr int kStackDepth = 64;

struct RayInv {
    float ox, oy, oz, ix, iy, iz;
};

__device__ __forceinline__ float safe_inv(float d) {
    float r = 1.f / d;
    return isfinite(r) ? r : copysignf(1e30f, d);
}

// Three-input max / min (one instruction on sm_100 and later); NaN inputs
// are ignored as by fmaxf / fminf.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

constexpr float kSlabWiden = 2.f * 3.f * 0x1p-24f / (1.f - 3.f * 0x1p-24f);

// A ray for slab distances in one fused operation, t = plane * i + c with
// c = -(o * i) rounded.  Against (plane - o) * i, whose rounding is relative
// to t, the rounding of c adds u * |o * i| <= u * |t| + u * |plane * i|: the
// first part keeps the three roundings that kSlabWiden covers, the second
// moves the plane by u of its own magnitude, 2^-11 of the box's padding.
// Where o * i overflows while o is finite, c is NaN and the axis is ignored
// (fmax3 / fmin3 drop NaN), which keeps the box.
struct RayFma {
    float ix, iy, iz, cx, cy, cz;
};

__device__ __forceinline__ float slab_offset(float o, float i) {
    const float c = -__fmul_rn(o, i);
    return isinf(c) && !isinf(o) ? __int_as_float(0x7fffffff) : c;
}

__device__ __forceinline__ RayFma ray_fma(float4 o, float4 d) {
    const float ix = safe_inv(d.x), iy = safe_inv(d.y), iz = safe_inv(d.z);
    return RayFma{ix, iy, iz, slab_offset(o.x, ix), slab_offset(o.y, iy), slab_offset(o.z, iz)};
}

// Two fused multiply-adds in one instruction (sm_100 and later), each
// rounded as fmaf.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z, w;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// Elements k, k + 1 (k even) of eight floats held as two float4.
__device__ __forceinline__ float2 pair_of(const float4* v, int k) {
    const float4 q = v[k >> 2];
    return (k & 2) ? make_float2(q.z, q.w) : make_float2(q.x, q.y);
}

__device__ __forceinline__ bool slab(const RayInv& r, float lx, float hx, float ly, float hy,
                                     float lz, float hz, float tmin, float tmax, float* tnear) {
    float tx0 = (lx - r.ox) * r.ix, tx1 = (hx - r.ox) * r.ix;
    float ty0 = (ly - r.oy) * r.iy, ty1 = (hy - r.oy) * r.iy;
    float tz0 = (lz - r.oz) * r.iz, tz1 = (hz - r.oz) * r.iz;
    float tn = fmax3(fminf(tx0, tx1), fminf(ty0, ty1), fmaxf(fminf(tz0, tz1), tmin));
    float tf = fmin3(fmaxf(tx0, tx1), fmaxf(ty0, ty1), fminf(fmaxf(tz0, tz1), tmax));
    *tnear = tn;
    // tf + |tf| * 2*gamma(3): each t carries at most two roundings
    return tn <= fmaf(fabsf(tf), kSlabWiden, tf);
}

// The same test with fused distances, a box's two planes of an axis in one
// instruction.
__device__ __forceinline__ bool slab(const RayFma& r, float lx, float hx, float ly, float hy,
                                     float lz, float hz, float tmin, float tmax, float* tnear) {
    const float2 tx = fma2(make_float2(lx, hx), make_float2(r.ix, r.ix), make_float2(r.cx, r.cx));
    const float2 ty = fma2(make_float2(ly, hy), make_float2(r.iy, r.iy), make_float2(r.cy, r.cy));
    const float2 tz = fma2(make_float2(lz, hz), make_float2(r.iz, r.iz), make_float2(r.cz, r.cz));
    const float tn = fmax3(fminf(tx.x, tx.y), fminf(ty.x, ty.y), fmaxf(fminf(tz.x, tz.y), tmin));
    const float tf = fmin3(fmaxf(tx.x, tx.y), fmaxf(ty.x, ty.y), fminf(fmaxf(tz.x, tz.y), tmax));
    *tnear = tn;
    return tn <= fmaf(fabsf(tf), kSlabWiden, tf);
}

// A node in two 32-byte loads (sm_100 and later; nodes start on multiples of
// their 64 bytes) instead of four of 16: the ordered walk of 921,600 rays 642
// -> 635 us, direct lighting's packets 870 -> 867 us a frame.
__device__ __forceinline__ BvhNode load_node(const BvhNode* p) {
    BvhNode n;
    float4 a;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.n0.x), "=f"(n.n0.y), "=f"(n.n0.z), "=f"(n.n0.w), "=f"(n.n1.x), "=f"(n.n1.y), "=f"(n.n1.z), "=f"(n.n1.w)
        : "l"(p));
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.n2.x), "=f"(n.n2.y), "=f"(n.n2.z), "=f"(n.n2.w), "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
        : "l"(reinterpret_cast<const char*>(p) + 32));
    n.n3 = make_int4(__float_as_int(a.x), __float_as_int(a.y), __float_as_int(a.z), __float_as_int(a.w));
    return n;
}

// The walk's stack.  PACK: one 8-byte entry (one local load per pop) when
// the scene allows it: a child reference, with a leaf's record start (below
// 2^24) and triangle count (below 128) packed into one negative word, and
// the entry distance.  Otherwise reference, count and distance in three
// arrays.
template <bool PACK>
struct WalkStack;

template <>
struct WalkStack<true> {
    int2 e[kStackDepth];
    __device__ __forceinline__ void put(int i, int32_t ref, int32_t cnt, float t) {
        const int32_t v = ref >= 0 ? ref : (int32_t)(0x80000000u | ((uint32_t)cnt << 24) | (uint32_t)(~ref));
        e[i] = make_int2(v, __float_as_int(t));
    }
    // entry i: its distance, and (reference, count) when it is taken
    __device__ __forceinline__ float get(int i, int32_t* ref, int32_t* cnt) const {
        const int2 v = e[i];
        if (v.x >= 0) {
            *ref = v.x;
            *cnt = 0;
        } else {
            *ref = ~(int32_t)((uint32_t)v.x & 0xffffffu);
            *cnt = (int32_t)(((uint32_t)v.x >> 24) & 0x7fu);
        }
        return __int_as_float(v.y);
    }
};

template <>
struct WalkStack<false> {
    int32_t r[kStackDepth], c[kStackDepth];
    float tt[kStackDepth];
    __device__ __forceinline__ void put(int i, int32_t ref, int32_t cnt, float t) {
        r[i] = ref;
        c[i] = cnt;
        tt[i] = t;
    }
    __device__ __forceinline__ float get(int i, int32_t* ref, int32_t* cnt) const {
        *ref = r[i];
        *cnt = c[i];
        return tt[i];
    }
};

struct WalkHit {
    float t, b1, b2;
    int32_t prim;
};

// A ray's state before its first hit.  h.t may be NaN (a maxt, or the distance
// of a hit whose products over- or underflowed), which rejects nothing in
// pbrt's test: the walks keep what is not beyond it, !(te > h.t).  (Making it
// +inf here spills more: 64 scenes 5,160 -> 5,274 us.)
__device__ __forceinline__ WalkHit unhit(float4 d) { return WalkHit{d.w, 0.f, 0.f, -1}; }

// The exact test of record `rec` and its effect on the hit; returns true when
// an any-hit query is done.
template <bool ANY, bool STATS>
__device__ __forceinline__ bool test_exact(const TriRec* __restrict__ tris, int32_t rec, float4 o, float4 d,
                                           WalkHit& h, WorkCount& wc) {
    const TriRec tr = tris[rec];
    float tt, u1, u2;
    if (STATS) wc.exact++;
    if (!pbg_exact_rec(tr, o, d, h.t, &tt, &u1, &u2)) return false;
    if (STATS) wc.hit++;
    const int32_t id = __float_as_int(tr.c.w);
    if (ANY) {
        h.prim = id;
        return true;
    }
    if (tt < h.t || id > h.prim) {
        h.t = tt;
        h.prim = id;
        h.b1 = u1;
        h.b2 = u2;
    }
    return false;
}

// Tests records [start, start + cnt); returns true when an any-hit query is
// done.  A record that passes the filter waits for the next that does, or for
// the last record: few of the warp's rays pass at one record, and its exact
// test takes as long for one ray as for 32 (ordered walk 666 -> 642 us, 500
// picking rays 19.2 -> 18.4).  HOLD false: each at once, for the walk of one
// thread per ray, whose lanes are seldom in a leaf together (307,200 bounce rays
// on 1,024,000 triangles 512 -> 469 us, camera rays 392 -> 369).
template <bool ANY, bool STATS, bool HOLD = true>
__device__ __forceinline__ bool test_run(const TriRec* __restrict__ tris, int32_t start, int32_t cnt,
                                         float4 o, float4 d, float nd, WalkHit& h, WorkCount& wc) {
    int32_t pend = -1;
    for (int32_t k = 0; k < cnt; ++k) {
        if (STATS) wc.filt++;
        if (!pbg_filter(tris[start + k], o, d, nd, h.t, STATS ? &wc.filt2 : nullptr)) continue;
        if (!HOLD) {
            if (test_exact<ANY, STATS>(tris, start + k, o, d, h, wc)) return true;
            continue;
        }
        if (pend >= 0 && test_exact<ANY, STATS>(tris, pend, o, d, h, wc)) return true;
        pend = start + k;
    }
    return pend >= 0 && test_exact<ANY, STATS>(tris, pend, o, d, h, wc);
}

// The walk.  h.t starts at the ray's maxt and h.prim at -1.  ORDERED: the
// child reference `first_ref` (a cluster the learned model picked, with leaf
// count first_cnt) is walked first and skipped later; INT32_MIN = none.
// Returns false if the private stack overflowed (the result may then miss
// hits; the caller raises the overflow status).
template <bool ANY, bool STATS, bool ORDERED>
__device__ __forceinline__ bool bvh_walk(const BvhNode* __restrict__ nodes, const TriRec* __restrict__ tris,
                                         int32_t unculled, float4 o, float4 d, int32_t first_ref,
                                         int32_t first_cnt, WalkHit& h, WorkCount& wc) {
    const float nd = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    const RayInv ri{o.x, o.y, o.z, safe_inv(d.x), safe_inv(d.y), safe_inv(d.z)};
    bool done = unculled > 0 && test_run<ANY, STATS, false>(tris, 0, unculled, o, d, nd, h, wc);
    int2 stack[kStackDepth];  // (inner node, entry distance bits): one 8-byte entry
    int sp = 0;
    int32_t node = 0;
    bool ok = true;
    const int32_t skip = ORDERED ? first_ref : INT32_MIN;
    if (ORDERED && !done && first_ref != INT32_MIN) {
        if (first_ref < 0) {
            if (STATS) wc.leaf++;
            done = test_run<ANY, STATS, false>(tris, ~first_ref, first_cnt, o, d, nd, h, wc);
        } else {
            stack[sp] = make_int2(0, __float_as_int(-INFINITY));  // resume at the root afterwards
            ++sp;
            node = first_ref;
        }
    }
    while (!done) {
        const BvhNode nd_ = nodes[node];
        if (STATS) wc.node += 2;
        float tn0, tn1;
        bool h0 = slab(ri, nd_.n0.x, nd_.n0.y, nd_.n0.z, nd_.n0.w, nd_.n2.x, nd_.n2.y, o.w, h.t, &tn0);
        bool h1 = slab(ri, nd_.n1.x, nd_.n1.y, nd_.n1.z, nd_.n1.w, nd_.n2.z, nd_.n2.w, o.w, h.t, &tn1);
        const int32_t c0 = nd_.n3.x, c1 = nd_.n3.y;
        if (ORDERED) {  // the predicted cluster has been walked already
            h0 = h0 && c0 != skip;
            h1 = h1 && c1 != skip;
        }
        // Leaf children are tested at once, nearer one first.
        const bool swap = h0 && h1 && tn1 < tn0;
        for (int q = 0; q < 2 && !done; ++q) {
            const int side = swap ? 1 - q : q;
            const bool hh = side == 0 ? h0 : h1;
            const int32_t c = side == 0 ? c0 : c1;
            if (!hh || c >= 0) continue;
            if (STATS) wc.leaf++;
            done = test_run<ANY, STATS, false>(tris, ~c, side == 0 ? nd_.n3.z : nd_.n3.w, o, d, nd, h, wc);
        }
        if (done) break;
        h0 = h0 && c0 >= 0;
        h1 = h1 && c1 >= 0;
        if (h0 && h1) {
            const bool first0 = tn0 <= tn1;
            if (sp < kStackDepth) {
                stack[sp] = make_int2(first0 ? c1 : c0, __float_as_int(first0 ? tn1 : tn0));
                ++sp;
            } else {
                ok = false;
            }
            node = first0 ? c0 : c1;
            continue;
        }
        if (h0 || h1) {
            node = h0 ? c0 : c1;
            continue;
        }
        bool found = false;
        while (sp > 0) {
            --sp;
            const int2 e = stack[sp];
            if (!(__int_as_float(e.y) > h.t)) {
                node = e.x;
                found = true;
                break;
            }
        }
        if (!found) break;
    }
    return ok;
}

#endif  // __CUDACC__

}  // namespace pbg
