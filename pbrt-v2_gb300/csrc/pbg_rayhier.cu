// pbg_rayhier.cu -- Accelerator "rayhierarchy": a hierarchy over the rays of
// each batch, rebuilt per call, traversed by the triangles.
//
// Reference: RayHieararchy (accelerators/rayhierarchy.cpp:375-1326) builds a
// quadtree over the batch's 2-D ray image -- leaves of chunkX x chunkY rays
// bounded by a 6-D box (origin AABB + direction AABB, bin/cl/rayhconstruct6DB.cl),
// parents by 2x2 merges (levelConstruct6DB.cl) -- and launches one thread per
// triangle that walks the tree with a global-memory stack
// (intersection6DB.cl:6-120), racing on tHit and repairing the races with
// extra passes (yetAnotherIntersection6DB.cl).
//
// Here:
//   build     rays ordered (pbg_rayorder.cu: the declared ray image in 2-D
//             Morton order, shadow batches along a 3-D Hilbert curve of their
//             origins, otherwise a 6-D Morton code) and gathered; a leaf is
//             32 consecutive rays (one warp builds it with shuffle
//             reductions); parents merge 4 children, up to the level the
//             descent is seeded at (no level above it is built).  A node is
//             bounded by an origin sphere (centre, radius), a direction cone
//             (unit axis, cos/sin of the half-angle) and the farthest reach
//             of its rays (max maxt*|d|).  A shadow batch whose origins and
//             validity repeat the previous batch's takes the kept order and
//             sorted origins at once; the comparison's answer is read with
//             the batch's closing status word and a batch whose origins moved
//             is traced again in a fresh order.
//   traverse  triangle records in clusters of 32 (SAH-style splits on whole
//             clusters, bvh_build.cpp), node test = "can any ray of the node
//             come within R of the triangle's or cluster's bounding sphere",
//             leaf test = the exact test per ray; the clusters walk the
//             levels level by level, seeded at the first level of at most
//             1,024 nodes; at the leaves'
//             parents a warp splits its cluster and tests the reaching
//             members against each leaf's rays directly; other split levels
//             group the (triangle, leaf) pairs by leaf first so a warp
//             loads a leaf's rays once for all its triangles.
//             Nearest hits merge through a 64-bit atomicMax on (t, index)
//             keys -- race-free by construction, no repair pass; a thread
//             reads a ray's current key first and filters with that t.
//             Nearest-hit batches take the final (cluster, leaves' parent)
//             pairs front to back (by distance from the parent's origin
//             ball) and cull with live reach bounds per leaf and parent.
//             Any-hit keeps one occlusion bit per ray (a 32-bit mask per
//             leaf) and skips leaves whose rays are all occluded.
#include <algorithm>
#include <functional>

#include "pbg_internal.h"
#include "pbg_count.cuh"
#include "pbg_tma.cuh"

namespace pbg {

int ray_sort(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
             const int32_t** perm, const uint32_t** sorted_keys, cudaStream_t st, int order);
int scan_counts(pbg_scene* s, uint32_t* a, int64_t m, cudaStream_t st);

constexpr int kLeafRays = 32;
constexpr int kFan = 4;
constexpr int kMaxLevels = 16;

struct __align__(16) RayNode {
    float4 a;  // origin sphere: centre.xyz, radius
    float4 b;  // cone axis.xyz, cos(half-angle)
    float4 c;  // sin(half-angle), reach = max maxt*|d|, count (int bits), spread (beam_spread)
};

struct Levels {
    int64_t off[kMaxLevels];
    int64_t cnt[kMaxLevels];
    int nlev;
};

__device__ __forceinline__ float round_up_rel(float x) { return fmaf(fabsf(x), 0x1p-20f, x) + 0x1p-126f; }

// ---------------------------------------------------------------- build

// An upper bound on |u - axis| over the unit directions u of a cone with
// cosine c (already lowered by its rounding), or +inf where a ray's length is
// extreme (beam_misses' bounds then do not hold).
constexpr float kPlainDir = 0x1p30f;
__device__ __forceinline__ float beam_spread(float c, bool plain) {
    return plain ? sqrtf(2.f * (1.f - c)) * (1.f + 0x1p-16f) : INFINITY;
}

// A batch of at most this many rays has launches and few long pairs to wait
// for: its leaf build zeroes the traversal's words, its finalize kernel
// publishes the status, its split tests take a leaf per warp while there are
// few pairs, and its other kernels fewer CTAs; larger batches use memsets, a
// kernel of its own and a pair per warp.  A camera batch and two shadow batches
// of 19,159 / 131,400 / 256,000 / 518,400 / 700,000 / 1,048,576 rays, us: on
// 12,000 triangles 249 / 500 / 529 / 625 / 682 / 654 in the first form, 300 / 536
// / 552 / 624 / 676 / 635 in the second, which meet at the line; on 181,250
// triangles 483 / 785 / 853 / 1,024 / 1,078 / 1,121 and 475 / 780 / 840 / 995 /
// 1,040 / 1,071.
constexpr int64_t kFewRays = 1 << 19;
// CTAs per SM of the level kernels where tune.rh_grid has none: 12 for small
// batches (of 4, 12, 32: 175, 172, 177 us at 19,159 rays), 32 for others (best
// of 4, 8, 16, 32 on the terrain frame).
bool rh_small_batch(int64_t n) { return n <= kFewRays; }
int rh_default_grid(bool small) { return small ? 12 : 32; }

// Words of device memory that a batch starts from zero (its keys or
// occlusion bits, counters, bounds).
constexpr int kZeroRanges = 6;
struct ZeroWords {
    uint32_t* p[kZeroRanges] = {};
    int64_t n[kZeroRanges] = {};
    int count = 0;
    void add(void* ptr, size_t bytes) {  // a multiple of 4 bytes
        p[count] = (uint32_t*)ptr;
        n[count++] = (int64_t)(bytes / 4);
    }
};

// The least / greatest of the warp's values, NaN ignored as by fminf / fmaxf
// (one instruction, sm_100 and later, for ten of a shuffle tree).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// One warp per leaf of 32 sorted rays; the warp also gathers its rays into
// sorted order (so, sd) for the leaf tests.
// keep_o: the batch leaves from the same origins (bit for bit, mint
// included) in the same order as the previous one, whose sorted origins and
// leaf spheres are still in so / leaves: only the directions are gathered
// and only the cones rebuilt.
template <bool ZERO>
__global__ void leaf_build_kernel(const float4* __restrict__ ro, const float4* __restrict__ rd,
                                  const int32_t* __restrict__ perm, float4* __restrict__ so,
                                  float4* __restrict__ sd, const uint32_t* __restrict__ skeys, int64_t n,
                                  int64_t nleaf, RayNode* __restrict__ leaves, bool keep_o, const ZeroWords zero) {
    for (int k = 0; ZERO && k < zero.count; ++k)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < zero.n[k];
             i += (int64_t)gridDim.x * blockDim.x)
            zero.p[k][i] = 0u;
    const int64_t leaf = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (leaf >= nleaf) return;
    const int64_t i = leaf * kLeafRays + lane;
    const bool ok = i < n && skeys[i] != 0xffffffffu;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
    if (ok) {  // invalid rays sort last and are never read back: not gathered
        const int32_t src = perm[i];
        d = rd[src];
        sd[i] = d;
        if (!keep_o) {
            o = ro[src];
            so[i] = o;
        }
    }
    const unsigned full = 0xffffffffu;
    const int count = __popc(__ballot_sync(full, ok));
    float lo[3] = {ok ? o.x : INFINITY, ok ? o.y : INFINITY, ok ? o.z : INFINITY};
    float hi[3] = {ok ? o.x : -INFINITY, ok ? o.y : -INFINITY, ok ? o.z : -INFINITY};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = warp_min(lo[a]);
        hi[a] = warp_max(hi[a]);
    }
    const float len = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    const float il = len > 0.f ? 1.f / len : 0.f;
    float nx = d.x * il, ny = d.y * il, nz = d.z * il;
    float sx = ok ? nx : 0.f, sy = ok ? ny : 0.f, sz = ok ? nz : 0.f;
    float reach = ok ? d.w * len * (1.f + 0x1p-20f) : 0.f;
    if (ok && !(reach == reach)) reach = INFINITY;  // 0 * inf
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        sx += __shfl_xor_sync(full, sx, off);
        sy += __shfl_xor_sync(full, sy, off);
        sz += __shfl_xor_sync(full, sz, off);
    }
    reach = warp_max(reach);
    const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
    float dist = ok ? sqrtf((o.x - cx) * (o.x - cx) + (o.y - cy) * (o.y - cy) + (o.z - cz) * (o.z - cz)) : 0.f;
    const float sl = sqrtf(sx * sx + sy * sy + sz * sz);
    float ax = 0.f, ay = 0.f, az = 1.f;
    bool axis_ok = sl > 1e-3f * (float)(count > 0 ? count : 1);
    if (axis_ok) {
        ax = sx / sl;
        ay = sy / sl;
        az = sz / sl;
    }
    float cosv = ok ? (axis_ok ? ax * nx + ay * ny + az * nz : -1.f) : 2.f;
    if (ok && !(len > 0.f && isfinite(len))) cosv = -1.f;
    const bool plain = __all_sync(full, !ok || (len >= 1.f / kPlainDir && len <= kPlainDir));
    dist = warp_max(dist);
    cosv = warp_min(cosv);
    if (lane == 0) {
        RayNode nd;
        if (count == 0) {
            nd.a = make_float4(0.f, 0.f, 0.f, 0.f);
            nd.b = make_float4(0.f, 0.f, 1.f, 1.f);
            nd.c = make_float4(0.f, 0.f, __int_as_float(0), 0.f);
        } else {
            // Margins: 2^-20 relative on the radius, 2^-18 on the cone cosine.
            const float ro_ = round_up_rel(dist);
            float c = fmaxf(cosv - 0x1p-18f, -1.f);
            if (c > 1.f) c = 1.f;
            const float s = fminf(sqrtf(fmaxf(0.f, 1.f - c * c)) + 0x1p-18f, 1.f);
            nd.a = keep_o ? leaves[leaf].a : make_float4(cx, cy, cz, ro_);
            nd.b = make_float4(ax, ay, az, c);
            nd.c = make_float4(s, reach, __int_as_float(count), beam_spread(c, plain));
        }
        leaves[leaf] = nd;
    }
}

// Parent j merges children kFan*j .. kFan*j+kFan-1.
__device__ __forceinline__ void build_parent(const RayNode* __restrict__ child, int64_t nchild,
                                             RayNode* __restrict__ parent, int64_t j) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    float sx = 0.f, sy = 0.f, sz = 0.f, reach = 0.f;
    int count = 0;
    RayNode ch[kFan];
    int nk = 0;
    for (int k = 0; k < kFan; ++k) {
        const int64_t c = kFan * j + k;
        if (c >= nchild) break;
        ch[nk] = child[c];
        const int cc = __float_as_int(ch[nk].c.z);
        if (cc == 0) continue;
        const float4 a = ch[nk].a;
        lo[0] = fminf(lo[0], a.x - a.w); hi[0] = fmaxf(hi[0], a.x + a.w);
        lo[1] = fminf(lo[1], a.y - a.w); hi[1] = fmaxf(hi[1], a.y + a.w);
        lo[2] = fminf(lo[2], a.z - a.w); hi[2] = fmaxf(hi[2], a.z + a.w);
        sx += ch[nk].b.x * cc;
        sy += ch[nk].b.y * cc;
        sz += ch[nk].b.z * cc;
        reach = fmaxf(reach, ch[nk].c.y);
        count += cc;
        ++nk;
    }
    RayNode nd;
    if (count == 0) {
        nd.a = make_float4(0.f, 0.f, 0.f, 0.f);
        nd.b = make_float4(0.f, 0.f, 1.f, 1.f);
        nd.c = make_float4(0.f, 0.f, __int_as_float(0), 0.f);
        parent[j] = nd;
        return;
    }
    const float cx = 0.5f * (lo[0] + hi[0]), cy = 0.5f * (lo[1] + hi[1]), cz = 0.5f * (lo[2] + hi[2]);
    const float sl = sqrtf(sx * sx + sy * sy + sz * sz);
    const bool axis_ok = sl > 1e-3f * count;
    float ax = 0.f, ay = 0.f, az = 1.f;
    if (axis_ok) {
        ax = sx / sl;
        ay = sy / sl;
        az = sz / sl;
    }
    float r = 0.f, cmin = 1.f;
    for (int k = 0; k < nk; ++k) {
        const float4 a = ch[k].a;
        const float dx = a.x - cx, dy = a.y - cy, dz = a.z - cz;
        r = fmaxf(r, sqrtf(dx * dx + dy * dy + dz * dz) + a.w);
        // cos(angle(axis, child axis) + child half-angle)
        const float ca = axis_ok ? fminf(1.f, fmaxf(-1.f, ax * ch[k].b.x + ay * ch[k].b.y + az * ch[k].b.z)) : -1.f;
        const float sa = sqrtf(fmaxf(0.f, 1.f - ca * ca));
        const float cb = ch[k].b.w, sb = ch[k].c.x;
        // alpha + beta >= pi  <=>  cos(alpha) <= -cos(beta) (alpha, beta in [0, pi])
        const float csum = (ca <= -cb) ? -1.f : ca * cb - sa * sb;
        cmin = fminf(cmin, csum);
    }
    const float c = fmaxf(cmin - 0x1p-18f, -1.f);
    const float s = fminf(sqrtf(fmaxf(0.f, 1.f - c * c)) + 0x1p-18f, 1.f);
    nd.a = make_float4(cx, cy, cz, round_up_rel(r));
    nd.b = make_float4(ax, ay, az, c);
    nd.c = make_float4(s, reach, __int_as_float(count), 0.f);
    parent[j] = nd;
}

// Levels l0 + 1 .. l1 of the subtrees above groups of kFan^(l1 - l0) nodes
// of level l0: CTA g builds its subtree level by level (children written
// by the same CTA in the previous round), so five levels take one launch.
constexpr int kLevelsPerLaunch = 5;

__global__ void __launch_bounds__(256) level_build_multi_kernel(RayNode* __restrict__ nodes, Levels lv,
                                                                 int l0, int l1) {
    const int64_t span0 = 1ll << (2 * (l1 - l0));
    for (int l = l0 + 1; l <= l1; ++l) {
        const int64_t span = span0 >> (2 * (l - l0));
        const int64_t first = (int64_t)blockIdx.x * span;
        const int64_t last = min(first + span, lv.cnt[l]);
        for (int64_t j = first + threadIdx.x; j < last; j += blockDim.x)
            build_parent(nodes + lv.off[l - 1], lv.cnt[l - 1], nodes + lv.off[l], j);
        __syncthreads();
    }
}

// --------------------------------------------------------------- traverse

// Can a ray of node `nd` pass within reach of the sphere (c, r)?  r already
// holds the triangle's padding.  Conservative in float: every comparison
// carries a relative margin.
__device__ __forceinline__ bool node_hits_sphere(const RayNode& nd, float4 sph) {
    const float vx = sph.x - nd.a.x, vy = sph.y - nd.a.y, vz = sph.z - nd.a.z;
    const float dist2 = vx * vx + vy * vy + vz * vz;
    // Square roots by the hardware reciprocal square root (error a few ulp):
    // dist_lo / dist_hi bracket the distance by 2^-18, far inside the test's
    // own margins; 0 and inf give NaN, which keeps the pair.
    const float dist = dist2 * rsqrtf(dist2);
    const float dist_lo = dist * (1.f - 0x1p-18f), dist_hi = dist * (1.f + 0x1p-18f);
    // slop of pbrt's float test grows with the distance from the ray origin
    const float R = sph.w + nd.a.w + dist_hi * 0x1p-12f;
    if (!(dist_lo > R)) return true;  // overlapping (or NaN): keep
    if (dist_lo - R > nd.c.y * (1.f + 0x1p-18f)) return false;  // beyond every ray's maxt
    // With the sphere seen under half-angle beta (sin = R/dist, cos = q/dist)
    // and the cone's half-angle theta, the test is angle(axis, v) <= theta +
    // beta, i.e. axis.v >= dist cos(theta + beta) = cos(theta) q - sin(theta) R,
    // scaled by dist so that no division is needed.
    const float q2 = (dist_hi - R) * (dist_hi + R);  // > 0 here
    const float q = q2 * rsqrtf(q2);
    const float cth = nd.b.w, sth = nd.c.x;
    if (cth * dist <= -q) return true;  // cone half-angle + sphere angle >= pi
    const float dotv = vx * nd.b.x + vy * nd.b.y + vz * nd.b.z;
    return dotv >= cth * q - sth * R - 0x1p-16f * dist_hi;
}

// Whether every ray of a leaf certainly misses the triangle: pbrt's test,
// s1 = d x e2, div = s1.e1, b1 = (v.s1) / div, b2 = (d.(v x e1)) / div with
// v = o - p1, over all origins within r of the leaf's centre and unit
// directions u within the spread of its axis a.  With w = centre - p1, for
// every ray
//   div / |d|          = u.(e2 x e1)  is within spread |e2 x e1| of a.(e2 x e1),
//   (b1 div) / |d|     = u.(e2 x v)   within spread |e2 x w| + |e2| r of a.(e2 x w),
//   (b2 div) / |d|     = u.(v x e1)   within spread |w x e1| + |e1| r of a.(w x e1),
//   ((b1 + b2 - 1) div) / |d|, the sum of the last two less the first,
//                      = u.((e2 - e1) x (v - e1)), its bound likewise.
// So the triangle is missed where the divisor's sign is certain and b1 < 0,
// b2 < 0 or b1 + b2 > 1 for all of them.  2^-17 of the lengths covers pbrt's
// rounding of each product (9.1 u with u = 2^-24, see pbg_exact.cuh), the
// rounding here and that of b1, b2 and their sum; edges, distances (a tiny one
// too: the origins at a vertex) and directions of extreme size, where products
// may overflow or underflow, are never missed, and a NaN anywhere keeps the
// triangle.
__device__ __forceinline__ float rough_len(float x, float y, float z) {
    const float l2 = x * x + y * y + z * z;
    return l2 * rsqrtf(l2);  // within 2^-20, inside the spread's own margin
}
// Only the rays of a narrow leaf have much in common: in a leaf whose cone is
// wider than kNarrow the beam misses next to nothing, and so many members pass
// the filter for some ray that holding exact tests back only adds votes.
// Bounds of 0.06 to 1 do the same for camera rays (385 us for 518,400 on 181,250
// triangles, 402 with no leaf narrow); 200,000 incoherent rays there take 21.3
// ms with every leaf narrow, 18.8 so, 256,036 bounce rays 41.8 and 37.8.
constexpr float kNarrow = 0.25f;
__device__ __forceinline__ bool beam_misses(const RayNode& nd, const TriRec& tr) {
    constexpr float kTol = 0x1p-17f, kBig = 0x1p29f;
    const float e1x = tr.b.x, e1y = tr.b.y, e1z = tr.b.z, e2x = tr.c.x, e2y = tr.c.y, e2z = tr.c.z;
    const float ne1 = tr.a.w, ne2 = tr.b.w, r = nd.a.w, spread = nd.c.w;
    const float wx = nd.a.x - tr.a.x, wy = nd.a.y - tr.a.y, wz = nd.a.z - tr.a.z;
    const float nw = fabsf(wx) + fabsf(wy) + fabsf(wz) + r;
    const float mx = fmaf(e2y, e1z, -(e2z * e1y)), my = fmaf(e2z, e1x, -(e2x * e1z)), mz = fmaf(e2x, e1y, -(e2y * e1x));
    const float q1x = fmaf(e2y, wz, -(e2z * wy)), q1y = fmaf(e2z, wx, -(e2x * wz)), q1z = fmaf(e2x, wy, -(e2y * wx));
    const float q2x = fmaf(wy, e1z, -(wz * e1y)), q2y = fmaf(wz, e1x, -(wx * e1z)), q2z = fmaf(wx, e1y, -(wy * e1x));
    const float ax = nd.b.x, ay = nd.b.y, az = nd.b.z;
    const float div = ax * mx + ay * my + az * mz;
    const float n1 = flip_sign(ax * q1x + ay * q1y + az * q1z, div), n2 = flip_sign(ax * q2x + ay * q2y + az * q2z, div);
    const float D = fabsf(div), ee = kTol * ne1 * ne2, rt = fmaf(kTol, nw, r);
    const bool certain = D > fmaf(spread, rough_len(mx, my, mz), ee) && fminf(fminf(ne1, ne2), nw) >= 1.f / kBig &&
                         fmaxf(fmaxf(ne1, ne2), nw) <= kBig;
    const float n3 = ne1 + ne2;
    return certain && (n1 < -fmaf(spread, rough_len(q1x, q1y, q1z), ne2 * rt) ||
                       n2 < -fmaf(spread, rough_len(q2x, q2y, q2z), ne1 * rt) ||
                       n1 + n2 - D > fmaf(spread, rough_len(q1x + q2x - mx, q1y + q2y - my, q1z + q2z - mz),
                                          fmaf(kTol * n3, nw, fmaf(fabsf(e2x - e1x) + fabsf(e2y - e1y) + fabsf(e2z - e1z), r, ee))));
}

// A (triangle record, node) pair that passed its node test.
struct Pair {
    int32_t tri;
    int32_t node;
};

// Appends up to kFan items per thread with one atomic per warp; items past
// the capacity are dropped and flagged (the host then reruns with smaller
// triangle groups).  Every lane of the warp must call it.
__device__ __forceinline__ void warp_append(const Pair* items, int k, Pair* q, uint32_t* count,
                                            uint32_t cap, int* status) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int incl = k;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(full, incl, off);
        if (lane >= off) incl += y;
    }
    const int total = __shfl_sync(full, incl, 31);
    uint32_t base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(count, (uint32_t)total);
    base = __shfl_sync(full, base, 31);
    const uint32_t start = base + (uint32_t)(incl - k);
    for (int j = 0; j < k; ++j) {
        const uint32_t pos = start + (uint32_t)j;
        if (pos < cap) q[pos] = items[j];
    }
    if (lane == 31 && total > 0 && base + (uint32_t)total > cap) atomicAdd(&status[kStatusOverflow], 1);
}

// Level-synchronous descent.  Pairs of level `lvl` (already tested) produce
// the pairs of their children that pass.  The descent is seeded at a level
// of at most kSeedNodes nodes: every (cluster or triangle in [t0, t1), node)
// pair there is tested directly, which replaces the launches of the nearly
// empty levels above it.
// 1,024 nodes measured best: frames of 100,000 rays 347 us (256) / 327 / 327
// (2,048), 700,000 rays 1,430 / 1,397 / 1,455, 1024 x 1024 x 4 samples 2,850 /
// 2,836 / 2,966.
constexpr int64_t kSeedNodes = 1024;

template <bool STATS>
__global__ void __launch_bounds__(256)
    rh_seed_kernel(const float4* __restrict__ spheres, int32_t t0, int32_t t1,
                   const RayNode* __restrict__ level_nodes, int64_t nnodes, Pair* __restrict__ out,
                   uint32_t* count, uint32_t cap, int* status, unsigned long long* wc) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t total = (int64_t)(t1 - t0) * nnodes;
    WorkCount c_;
    // this thread's (triangle or cluster, node), kept up by addition
    const int64_t start = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t step_t = (int32_t)(stride / nnodes), step_n = (int32_t)(stride % nnodes);
    int32_t t = t0 + (int32_t)(start / nnodes), node = (int32_t)(start % nnodes);
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < total; base += stride) {
        const int64_t i = base + threadIdx.x;
        Pair item[1];
        int k = 0;
        if (i < total) {
            const RayNode nd = level_nodes[node];
            if (__float_as_int(nd.c.z) > 0) {
                if (STATS) c_.node++;
                if (node_hits_sphere(nd, spheres[t])) item[k++] = Pair{t, node};
            }
        }
        warp_append(item, k, out, count, cap, status);
        t += step_t;
        node += step_n;
        if (node >= nnodes) {
            node -= (int32_t)nnodes;
            ++t;
        }
    }
    if (STATS) c_.flush(wc);
}

template <bool STATS>
__global__ void __launch_bounds__(256)
    rh_expand_kernel(const float4* __restrict__ spheres, const RayNode* __restrict__ child_nodes,
                     int64_t nchild, const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                     Pair* __restrict__ out, uint32_t* out_count, uint32_t cap, int* status,
                     unsigned long long* wc) {
    const uint32_t nin = min(*in_count, cap);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    WorkCount c_;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nin; base += stride) {
        const int64_t i = base + threadIdx.x;
        Pair item[kFan];
        int k = 0;
        if (i < nin) {
            const Pair p = in[i];
            const float4 sph = spheres[p.tri];
            const int64_t first = (int64_t)p.node * kFan;
            const int64_t last = min(first + kFan, nchild);
            for (int64_t c = first; c < last; ++c) {
                const RayNode nd = child_nodes[c];
                if (__float_as_int(nd.c.z) == 0) continue;
                if (STATS) c_.node++;
                if (node_hits_sphere(nd, sph)) item[k++] = Pair{p.tri, (int32_t)c};
            }
        }
        warp_append(item, k, out, out_count, cap, status);
    }
    if (STATS) c_.flush(wc);
}

// (cluster, node) pairs -> (triangle, node) pairs for the cluster's members
// in [t0, t1) whose own sphere passes the same node test: one warp per pair,
// lane j = member j.
template <bool STATS>
__global__ void __launch_bounds__(256)
    rh_split_kernel(const float4* __restrict__ spheres, int32_t t0, int32_t t1,
                    const RayNode* __restrict__ level_nodes, const Pair* __restrict__ in,
                    const uint32_t* __restrict__ in_count, Pair* __restrict__ out, uint32_t* out_count,
                    uint32_t cap, int* status, unsigned long long* wc) {
    const uint32_t nin = min(*in_count, cap);
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    WorkCount c_;
    // every lane of a warp runs the same number of iterations (warp_append)
    for (int64_t p = warp; p < nin; p += nwarps) {
        const Pair pr = in[p];
        const int64_t t = (int64_t)pr.tri * kClusterTris + lane;
        Pair item[1];
        int k = 0;
        if (t >= t0 && t < t1) {
            const RayNode nd = level_nodes[pr.node];
            if (STATS) c_.node++;
            if (node_hits_sphere(nd, spheres[t])) item[k++] = Pair{(int32_t)t, pr.node};
        }
        warp_append(item, k, out, out_count, cap, status);
    }
    if (STATS) c_.flush(wc);
}

// The last two levels and the leaf tests in one pass, no pair queue: one
// warp per (cluster, leaves' parent) pair.  Lane j first stands for member
// triangle j (parent test); the members that pass go side by side into shared
// memory, and every eight of them are tested against the kFan leaves at once,
// lane = (member, leaf).  Then, leaf by leaf, lane k stands for ray k of the
// leaf and puts the reaching members through the filter one after another; the
// exact test follows once for all rays.  A leaf's rays are loaded once per
// cluster that reaches it (from L2), instead of going through a written,
// counted, sorted and re-read list of (triangle, leaf) pairs.  Nearest:
// per-lane best key, atomicMax per leaf; any-hit: the leaf's occlusion bits
// are read first and set when a ray is blocked.
//
// Bound by instruction issue (86 % active, 20 of 32 lanes).  The frame of 4.2 M
// camera and 4 x 4.2 M shadow rays on 181,250 triangles, all five launches:
// 2,430 us before, 1,680 now.  Pairs differ so much in work that dealing them
// out by a fixed stride left a tail: any-hit 4 x 455 us, 386 from the counter.
// Exact tests held back: 386 -> 321.  Leaf tests by (member, leaf) and
// beam_misses: nearest 490 -> 440 and 656 -> 592 (both in narrow leaves only for
// nearest hits: kNarrow).
constexpr int kSplitWarps = 8;
constexpr int kSplitBlocks = 4;  // CTAs per SM, all resident: best of 4 (any-hit 1,283 us a frame), 5 (1,315), 6 (1,362)

// Nearest-hit batches also keep a live reach bound per leaf and per leaves'
// parent: an upper bound on maxt x |d| over the node's rays, where each
// ray's maxt has shrunk to its best hit so far (hits are only replaced by
// nearer ones, or by the higher index at equal t, which the node test's
// strict comparison keeps).  A member whose sphere lies wholly beyond the
// bound cannot become any of the node's nearest hits, so it is culled like
// one beyond the rays' own maxt.  Stored as 0x7f800000 - bits(bound), so
// zeroed memory reads +inf and atomicMax lowers the bound.
__device__ __forceinline__ float live_reach(const uint32_t* b) {
    return __uint_as_float(0x7f800000u - __ldcg(b));
}
__device__ __forceinline__ void lower_reach(uint32_t* b, float x) {
    x = (x == x) ? fmaxf(x, 0.f) : INFINITY;  // NaN reads as unbounded
    atomicMax(b, 0x7f800000u - __float_as_uint(x));
}

// The CTA's next task: from the lot of `deal` tasks that it took from the
// grid's counter last (s_lot: first task, tasks handed out); the warp that
// finds the lot just empty takes the next one, and the warps that come before
// it is back take single tasks.  Lots of 8 keep the grid's one counter out of
// the way (a task per atomic of the whole grid: 1.9 a nanosecond at most);
// with fewer than kDeal tasks to a warp, single ones leave no warp idle.
constexpr uint32_t kDeal = 8;

__device__ __forceinline__ uint32_t next_task(unsigned long long* s_lot, uint32_t* next, uint32_t deal) {
    const unsigned long long w = atomicAdd(s_lot, 1ull);
    const uint32_t k = (uint32_t)w;
    if (k < deal) return (uint32_t)(w >> 32) + k;
    if (k > deal) return atomicAdd(next, 1u);
    const uint32_t first = atomicAdd(next, deal);
    atomicExch(s_lot, ((unsigned long long)first << 32) | 1ull);
    return first;
}

// FEW (batches of at most kFewRays rays): with less than kByLeaf pairs to a
// warp, where the longest one is the kernel's time, a warp takes one leaf of a
// pair and tests the members against the parent again (19,159 camera and
// shadow rays on 12,000 triangles: 163 us, 194 by pairs).  With more of them
// that only adds work, and the parents' live bounds, which one leaf cannot
// lower, cull nothing: 19,159 bounce rays on 1,000,000 triangles 22.2 ms by
// leaves, 17.9 by pairs; 518,400 camera rays there 900 us, 588.  Lines at 0.3,
// 1, 4 and 12 pairs to a warp: 192 / 167 / 163 / 166 us for the first, 312 /
// 315 / 313 / 331 for 19,159 camera and shadow rays on 181,250 triangles.
constexpr uint32_t kByLeaf = 4;
template <bool ANY, bool STATS, bool FEW>
__global__ void __launch_bounds__(32 * kSplitWarps, kSplitBlocks)
    rh_split_test_kernel(const float4* __restrict__ spheres, const TriRec* __restrict__ tris, int32_t t0,
                         int32_t t1, const RayNode* __restrict__ level1, const RayNode* __restrict__ leaves,
                         int64_t nleaf, const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                         uint32_t cap, uint32_t* __restrict__ next, const float4* __restrict__ so,
                         const float4* __restrict__ sd,
                         unsigned long long* __restrict__ keys, uint32_t* __restrict__ leafmask,
                         uint32_t* __restrict__ leaf_reach, uint32_t* __restrict__ parent_reach,
                         const int* __restrict__ status, unsigned long long* wc) {
    __shared__ unsigned long long s_lot;
    __shared__ float4 s_rec[kSplitWarps][kClusterTris * 3];  // this warp's member records
    __shared__ float4 s_sph[kSplitWarps][kClusterTris];      // and spheres
    if (status[kStatusOverflow] != 0) return;  // pairs were dropped upstream: this attempt is rerun
    const unsigned full = 0xffffffffu;
    float4 *rec = s_rec[threadIdx.x >> 5], *msph = s_sph[threadIdx.x >> 5];
    const uint32_t nin = min(*in_count, cap);
    const int lane = threadIdx.x & 31;
    WorkCount c_;
    const bool by_leaf = FEW && nin < kByLeaf * kSplitWarps * gridDim.x;
    const int64_t ntask = by_leaf ? (int64_t)nin * kFan : nin;
    const uint32_t deal = ntask >= (int64_t)(kDeal * kSplitWarps) * gridDim.x ? kDeal : 1u;
    if (threadIdx.x == 0) s_lot = deal;
    __syncthreads();
    for (;;) {
        uint32_t task = 0;
        if (lane == 0) task = next_task(&s_lot, next, deal);
        task = __shfl_sync(full, task, 0);
        if (task >= ntask) break;
        const Pair pr = in[by_leaf ? task / kFan : task];
        const int64_t t = (int64_t)pr.tri * kClusterTris + lane;
        bool pass = false;
        float4 sph = make_float4(0.f, 0.f, 0.f, 0.f);
        float parent_now = INFINITY;
        if (t >= t0 && t < t1) {
            sph = spheres[t];
            if (STATS) c_.node++;
            RayNode pn = level1[pr.node];
            if (!ANY) {
                pn.c.y = fminf(pn.c.y, live_reach(parent_reach + pr.node));
                parent_now = pn.c.y;
            }
            pass = node_hits_sphere(pn, sph);
        }
        const unsigned members = __ballot_sync(full, pass);
        if (!members) continue;
        const int np = __popc(members);
        __syncwarp();  // the previous pair's records are no longer read
        if (pass) {  // the members that reach the parent, side by side
            const int k = __popc(members & ((1u << lane) - 1u));
            const TriRec own = tris[t];
            rec[3 * k] = own.a;
            rec[3 * k + 1] = own.b;
            rec[3 * k + 2] = own.c;
            msph[k] = sph;
        }
        __syncwarp();
        // Every eight of them against the kFan leaves at once: lane = (member,
        // leaf).  by_leaf: all against the task's leaf, lane = member.
        const int64_t first = (int64_t)pr.node * kFan;
        const int mine = by_leaf ? (int)(task % kFan) : lane % kFan;
        const int64_t my_leaf = first + mine;
        RayNode nd;
        nd.c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (my_leaf < nleaf) nd = leaves[my_leaf];
        const bool rays = __float_as_int(nd.c.z) > 0;
        if (!ANY && rays) nd.c.y = fminf(nd.c.y, live_reach(leaf_reach + my_leaf));
        unsigned mine_reached = 0;  // lane k: the leaves that member k reaches, one bit each
#pragma unroll 1
        for (int k0 = 0; k0 < np; k0 += by_leaf ? 32 : 32 / kFan) {
            const int k = k0 + (by_leaf ? lane : lane / kFan);
            bool reach = false;
            if (k < np && rays) {
                if (STATS) c_.node++;
                reach = node_hits_sphere(nd, msph[k]);
                if (!ANY && reach && nd.c.w <= kNarrow) {
                    TriRec own;
                    own.a = rec[3 * k];
                    own.b = rec[3 * k + 1];
                    own.c = rec[3 * k + 2];
                    reach = !beam_misses(nd, own);
                }
            }
            const unsigned b = __ballot_sync(full, reach);
            if (by_leaf)
                mine_reached = reach ? 1u << mine : 0u;
            else if (lane / (32 / kFan) == k0 / (32 / kFan))
                mine_reached = b >> (lane % (32 / kFan) * kFan) & ((1u << kFan) - 1u);
        }
        float parent_new = 0.f;  // max of the leaves' bounds after this pair
#pragma unroll 1
        for (int c = by_leaf ? mine : 0, c1 = by_leaf ? c + 1 : kFan; c < c1; ++c) {
            const int64_t leaf = first + c;
            unsigned m = __ballot_sync(full, mine_reached >> c & 1u);
            const float leaf_now = __shfl_sync(full, nd.c.y, c);  // by_leaf: every lane's leaf
            const int count = __shfl_sync(full, __float_as_int(nd.c.z), c);
            const bool narrow = ANY || __shfl_sync(full, nd.c.w, c) <= kNarrow;
            if (!m) {
                if (!ANY && count > 0) parent_new = fmaxf(parent_new, leaf_now);
                continue;
            }
            if (STATS && lane == 0) c_.leaf++;
            const int64_t r = leaf * kLeafRays + lane;
            bool active = lane < count;
            if (ANY && active) active = ((leafmask[leaf] >> lane) & 1u) == 0u;
            if (!__any_sync(full, active)) continue;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
            float nd1 = 0.f, maxt = 0.f;
            unsigned long long best = 0ull, start = 0ull;
            if (active) {
                o = so[r];
                d = sd[r];
                nd1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
                maxt = d.w;
                if (!ANY) {
                    start = best = keys[r];
                    if (start != 0ull) maxt = fminf(maxt, key_t(start));
                }
            }
            bool hit = false;
            // The exact test waits until the members are through the filter:
            // few rays pass for one member, and a warp's exact test takes as
            // long for one ray as for 32 (nearest hits: in narrow leaves).
            const auto exact = [&](int j, float* t) {
                TriRec tr;
                tr.a = rec[3 * j];
                tr.b = rec[3 * j + 1];
                tr.c = rec[3 * j + 2];
                float u1, u2;
                if (STATS) c_.exact++;
                const bool in = pbg_exact_rec(tr, o, d, maxt, t, &u1, &u2);
                if (STATS && in) c_.hit++;
                return in;
            };
            const auto filter = [&](int j) {
                TriRec tr;
                tr.a = rec[3 * j];
                tr.b = rec[3 * j + 1];
                tr.c = rec[3 * j + 2];
                if (STATS) c_.filt++;
                return pbg_filter(tr, o, d, nd1, maxt);
            };
            int pend = -1;  // this ray's member for the exact test
            if (ANY) {
                unsigned left = active ? m : 0u;  // this ray's members
                for (unsigned all = m; all; all = __reduce_or_sync(full, left)) {
                    pend = -1;
                    for (; all; all &= all - 1) {
                        const int j = __ffs(all) - 1;
                        if (!(left >> j & 1u)) continue;
                        if (filter(j)) {
                            pend = j;
                            left = 0u;
                        }
                    }
                    left = 0u;
                    float tt;
                    if (pend >= 0) {
                        hit = exact(pend, &tt);
                        if (!hit) left = m & ~((2u << pend) - 1u);  // rare: the members behind it
                    }
                }
            } else {
                const auto settle = [&]() {
                    float tt;
                    if (pend >= 0 && exact(pend, &tt)) {
                        const unsigned long long k = hit_key(tt, __float_as_int(rec[3 * pend + 2].w));
                        if (k > best) best = k;
                        maxt = tt;
                    }
                    pend = -1;
                };
                if (narrow) {
                    for (; m; m &= m - 1) {
                        const int j = __ffs(m) - 1;
                        const bool cand = active && filter(j);
                        if (__any_sync(full, cand && pend >= 0)) settle();
                        if (cand) pend = j;
                    }
                    settle();
                } else {
                    for (; m; m &= m - 1) {
                        pend = __ffs(m) - 1;
                        if (active && filter(pend)) settle();
                    }
                }
            }
            if (ANY) {
                if (hit) atomicOr(&leafmask[leaf], 1u << lane);
            } else {
                if (best > start) atomicMax(&keys[r], best);
                // the leaf's bound from its rays' maxt after this cluster
                // (2^-20 covers the rounding of |d|; lanes past count hold
                // no ray)
                const float len = sqrtf(fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)));
                float b = lane < count ? maxt * len * (1.f + 0x1p-20f) : 0.f;
                if (!(b == b)) b = INFINITY;
                b = warp_max(b);
                if (lane == 0 && b < leaf_now) lower_reach(leaf_reach + leaf, b);
                parent_new = fmaxf(parent_new, fminf(b, leaf_now));
            }
        }
        if (!ANY && !by_leaf && lane == 0 && parent_new < parent_now) lower_reach(parent_reach + pr.node, parent_new);
    }
    if (STATS) c_.flush(wc);
}

// Front-to-back order for the pairs of a nearest-hit batch: a counting sort
// of the (cluster, leaves' parent) pairs on the distance from the parent's
// origin ball to the cluster's sphere, so that the leaf tests, which take
// the pairs in queue order over time, meet the near clusters first and
// their hits lower the live reach bounds before the far clusters arrive.
// Buckets: the top bits of the float distance, 64 per octave.  The order
// only changes how much is culled, never a result.
constexpr int kOrderBuckets = 16384;

__device__ __forceinline__ uint32_t pair_bucket(float4 c, float4 ball) {
    const float dx = c.x - ball.x, dy = c.y - ball.y, dz = c.z - ball.z;
    float dist = sqrtf(dx * dx + dy * dy + dz * dz) - c.w - ball.w;
    if (!(dist > 0.f)) dist = 0.f;  // overlapping, or NaN
    return min(__float_as_uint(dist) >> 17, (uint32_t)kOrderBuckets - 1u);
}

__global__ void __launch_bounds__(256)
    rh_order_count_kernel(const float4* __restrict__ csph, const RayNode* __restrict__ level1,
                          const Pair* __restrict__ in, const uint32_t* __restrict__ in_count, uint32_t cap,
                          uint32_t* __restrict__ hist, const int* __restrict__ status) {
    if (status[kStatusOverflow] != 0) return;  // this attempt is rerun
    const uint32_t nin = min(*in_count, cap);
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nin; base += stride) {
        const int64_t i = base + threadIdx.x;
        const bool ok = i < nin;
        uint32_t key = (uint32_t)kOrderBuckets;
        if (ok) {
            const Pair pr = in[i];
            key = pair_bucket(csph[pr.tri], level1[pr.node].a);
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        if (ok && lane == __ffs(peers) - 1) atomicAdd(&hist[key], (uint32_t)__popc(peers));
    }
}

__global__ void __launch_bounds__(256)
    rh_order_scatter_kernel(const float4* __restrict__ csph, const RayNode* __restrict__ level1,
                            const Pair* __restrict__ in, const uint32_t* __restrict__ in_count, uint32_t cap,
                            uint32_t* __restrict__ cursor, Pair* __restrict__ out,
                            const int* __restrict__ status) {
    if (status[kStatusOverflow] != 0) return;
    const uint32_t nin = min(*in_count, cap);
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nin; base += stride) {
        const int64_t i = base + threadIdx.x;
        const bool ok = i < nin;
        Pair pr = Pair{0, 0};
        uint32_t key = (uint32_t)kOrderBuckets;
        if (ok) {
            pr = in[i];
            key = pair_bucket(csph[pr.tri], level1[pr.node].a);
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        uint32_t first = 0;
        if (ok && lane == leader) first = atomicAdd(&cursor[key], (uint32_t)__popc(peers));
        first = __shfl_sync(0xffffffffu, first, leader);
        const uint64_t dst = (uint64_t)first + __popc(peers & lt);
        if (ok && dst < nin) out[dst] = pr;
    }
}

// The final pairs grouped by leaf (a counting sort: count with ranks, scan,
// scatter), so that a leaf's 32 rays are loaded once for all the triangles
// that reach it instead of once per pair.
__global__ void rh_leaf_count_kernel(const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                                     uint32_t cap, uint32_t* __restrict__ leafcnt,
                                     uint32_t* __restrict__ rank) {
    const uint32_t nin = min(*in_count, cap);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nin; i += stride)
        rank[i] = atomicAdd(&leafcnt[in[i].node], 1u);
}

// After a queue overflow (pairs dropped; the host reruns the batch with more
// triangle groups) the counts and ranks no longer describe the queue, so the
// sort and the leaf tests of that attempt do nothing.
__global__ void rh_leaf_scatter_kernel(const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                                       uint32_t cap, const uint32_t* __restrict__ leafoff,
                                       const uint32_t* __restrict__ rank, Pair* __restrict__ out,
                                       const int* __restrict__ status) {
    if (status[kStatusOverflow] != 0) return;
    const uint32_t nin = min(*in_count, cap);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nin; i += stride) {
        const Pair p = in[i];
        const uint64_t dst = (uint64_t)leafoff[p.node] + rank[i];
        if (dst < nin) out[dst] = p;
    }
}

constexpr int kLeafChunk = 64;
constexpr int kLeafWarps = 8;  // warps per CTA of the leaf kernel

// One warp per chunk of kLeafChunk leaf-sorted pairs.  The chunk's pairs and
// triangle records are first staged in shared memory by the whole warp (so
// the loads overlap), then lane k tests ray k of the current leaf (loaded
// when the leaf changes) against each record.  Nearest: each lane keeps its
// best key and shrinks its maxt as it finds hits, merging with atomicMax
// when the leaf changes.  Any-hit: an occluded lane stops and sets its bit
// on leaving.
template <bool ANY, bool STATS>
__global__ void __launch_bounds__(32 * kLeafWarps)
    rh_leaf_sorted_kernel(const TriRec* __restrict__ tris, const RayNode* __restrict__ leaves,
                          const Pair* __restrict__ in, const uint32_t* __restrict__ in_count,
                          uint32_t cap, const float4* __restrict__ so, const float4* __restrict__ sd,
                          unsigned long long* __restrict__ keys, uint32_t* __restrict__ leafmask,
                          const int* __restrict__ status, unsigned long long* wc) {
    __shared__ float4 s_tri[kLeafWarps][kLeafChunk * 3];
    __shared__ Pair s_pair[kLeafWarps][kLeafChunk];
    if (status[kStatusOverflow] != 0) return;  // this attempt is rerun
    const uint32_t nin = min(*in_count, cap);
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float4* t4 = reinterpret_cast<const float4*>(tris);
    Pair* sp = s_pair[wib];
    float4* st4 = s_tri[wib];
    WorkCount c_;
    for (int64_t c0 = warp * kLeafChunk; c0 < nin; c0 += nwarps * kLeafChunk) {
        const int cnt = (int)min((int64_t)kLeafChunk, (int64_t)nin - c0);
        for (int j = lane; j < cnt; j += 32) sp[j] = in[c0 + j];
        __syncwarp();
        for (int j = lane; j < 3 * cnt; j += 32) st4[j] = t4[(int64_t)sp[j / 3].tri * 3 + j % 3];
        __syncwarp();
        int32_t leaf = -1;
        bool active = false, hit = false;
        int64_t r = 0;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
        float nd1 = 0.f, maxt = 0.f;
        unsigned long long best = 0ull, start = 0ull;
        for (int p = 0; p < cnt; ++p) {
            const Pair pr = sp[p];
            if (pr.node != leaf) {
                if (ANY) {
                    if (hit) atomicOr(&leafmask[leaf], 1u << lane);
                } else if (best > start) {
                    atomicMax(&keys[r], best);
                }
                leaf = pr.node;
                if (STATS && lane == 0) c_.leaf++;
                const int count = __float_as_int(leaves[leaf].c.z);
                r = (int64_t)leaf * kLeafRays + lane;
                active = lane < count;
                if (ANY && active) active = ((leafmask[leaf] >> lane) & 1u) == 0u;
                hit = false;
                if (active) {
                    o = so[r];
                    d = sd[r];
                    nd1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
                    maxt = d.w;
                    if (!ANY) {
                        start = best = keys[r];
                        if (start != 0ull) maxt = fminf(maxt, key_t(start));
                    }
                } else {
                    start = best = 0ull;
                }
            }
            if (!active) continue;
            TriRec tr;
            tr.a = st4[3 * p];
            tr.b = st4[3 * p + 1];
            tr.c = st4[3 * p + 2];
            if (STATS) c_.filt++;
            if (!pbg_filter(tr, o, d, nd1, maxt)) continue;
            float tt, u1, u2;
            if (STATS) c_.exact++;
            if (!pbg_exact_rec(tr, o, d, maxt, &tt, &u1, &u2)) continue;
            if (STATS) c_.hit++;
            if (ANY) {
                hit = true;
                active = false;
            } else {
                const unsigned long long k = hit_key(tt, __float_as_int(tr.c.w));
                if (k > best) best = k;
                maxt = tt;
            }
        }
        if (leaf >= 0) {
            if (ANY) {
                if (hit) atomicOr(&leafmask[leaf], 1u << lane);
            } else if (best > start) {
                atomicMax(&keys[r], best);
            }
        }
        __syncwarp();  // the next chunk overwrites this warp's staging
    }
    if (STATS) c_.flush(wc);
}

// The batch's status words to the host, from the finalize kernel's first
// thread: the kernel starts behind the leaf tests that set them.
struct Publication {
    const int* src = nullptr;
    int* dst = nullptr;
    int count = 0, seq = 0;
};
__device__ __forceinline__ void publish(const Publication& pub) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && pub.count > 0) publish_words(pub.src, pub.count, pub.dst, pub.seq);
}

// Sorted-order results back to the caller's order.
__global__ void rh_finalize_nearest(const TriRec* __restrict__ tris, const int32_t* __restrict__ pos,
                                    const float4* __restrict__ so, const float4* __restrict__ sd,
                                    const int32_t* __restrict__ perm,
                                    const unsigned long long* __restrict__ keys, int64_t n,
                                    int32_t* prim, float* t, float* b1, float* b2, const Publication pub) {
    publish(pub);
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t ray = perm[i];
    const unsigned long long k = keys[i];
    int32_t p = -1;
    float tt = 0.f, u1 = 0.f, u2 = 0.f;
    if (k != 0ull) {
        p = key_prim(k);
        const float4 o = so[i], d = sd[i];
        if (!pbg_exact_rec(tris[pos[p]], o, d, d.w, &tt, &u1, &u2)) {
            p = -1;
            tt = u1 = u2 = 0.f;
        }
    }
    prim[ray] = p;
    t[ray] = tt;
    b1[ray] = u1;
    b2[ray] = u2;
}

__global__ void rh_finalize_occluded(const int32_t* __restrict__ perm,
                                     const uint32_t* __restrict__ leafmask, int64_t n,
                                     uint8_t* occ, const Publication pub) {
    publish(pub);
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    occ[perm[i]] = (leafmask[i / kLeafRays] >> (i % kLeafRays)) & 1u;
}

// ------------------------------------------------------------------ host

// The levels the traversal reads: clusters split into triangles at level
// `split`, and the descent is seeded at `seed`, the lowest level of at most
// kSeedNodes (tune.rh_seed) nodes not below max(split, 1).  No level above the seed is
// read, so the build stops there.
struct Descent {
    int split, seed;
};
static Descent descent_levels(const pbg_scene* s, const Levels& lv, bool any) {
    const int top = lv.nlev - 1;
    // levels walked by 32-triangle clusters before they split into triangles
    // (default: down to the leaves' parents, the fastest split on the
    // terrain direct-lighting frame)
    int kcl = s->params.rh_cluster_levels;
    if (kcl == 0) kcl = std::max(1, top - 1);
    if (kcl < 0 || s->clusters.ptr == nullptr) kcl = 0;
    Descent d;
    d.split = std::max(0, top - kcl);
    d.seed = top;
    const int64_t seed_nodes = s->tune.rh_seed[any] > 0 ? s->tune.rh_seed[any] : kSeedNodes;
    while (d.seed > std::max(d.split, 1) && lv.cnt[d.seed - 1] <= seed_nodes) --d.seed;
    return d;
}

static int rh_workspace(pbg_scene* s, const Levels& lv, bool any, ZeroWords* zero);

// zero: what the caller needs zeroed, to which the traversal's words are added.
static int rh_build(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
                    const int32_t** perm, float4** so, float4** sd, Levels* lv, int order, ZeroWords* zero,
                    cudaStream_t st) {
    Work& w = s->work;
    const uint32_t* skeys = nullptr;
    const bool had_origins = w.sorted_origins_ok;
    w.sorted_origins_ok = false;  // set again once this hierarchy build has written them
    const void* before[2] = {w.ray_o2.ptr, w.nodes.ptr};
    int rc = ray_sort(s, o, d, valid, n, perm, &skeys, st, order);
    if (rc) return rc;
    if ((rc = ensure(w.ray_o2, (size_t)n * sizeof(float4))) ||
        (rc = ensure(w.ray_d2, (size_t)n * sizeof(float4))))
        return rc;
    *so = (float4*)w.ray_o2.ptr;
    *sd = (float4*)w.ray_d2.ptr;
    // levels: leaves of 32 rays, parents of 4 children, up to one root
    int64_t cnt = (n + kLeafRays - 1) / kLeafRays, total = 0;
    lv->nlev = 0;
    for (;;) {
        lv->off[lv->nlev] = total;
        lv->cnt[lv->nlev] = cnt;
        total += cnt;
        lv->nlev++;
        if (cnt <= 1 || lv->nlev == kMaxLevels) break;
        cnt = (cnt + kFan - 1) / kFan;
    }
    if ((rc = ensure(w.nodes, (size_t)total * sizeof(RayNode)))) return rc;
    RayNode* nodes = (RayNode*)w.nodes.ptr;
    const int64_t nleaf = lv->cnt[0];
    // the previous batch's sorted origins and leaf spheres still apply when
    // its order was reused and neither buffer moved
    const bool keep_o = order == kOrderOrigin && w.origin_reused && had_origins &&
                        before[0] == w.ray_o2.ptr && before[1] == w.nodes.ptr;
    if (s->ntri > 0 && (rc = rh_workspace(s, *lv, order == kOrderOrigin, zero))) return rc;
    const bool few = rh_small_batch(n);
    for (int k = 0; !few && k < zero->count; ++k) PBG_CUDA(cudaMemsetAsync(zero->p[k], 0, (size_t)zero->n[k] * 4, st));
    prof_begin(s, st);
    (few ? leaf_build_kernel<true> : leaf_build_kernel<false>)<<<(unsigned)((nleaf * 32 + 255) / 256), 256, 0, st>>>(
        o, d, *perm, *so, *sd, skeys, n, nleaf, nodes, keep_o, *zero);
    prof_end(s, st, kStageBuild, 1);
    // the levels above are never read (any-hit batches are the origin-ordered ones)
    const int built = descent_levels(s, *lv, order == kOrderOrigin).seed;
    for (int l0 = 0; l0 < built; l0 += kLevelsPerLaunch) {
        const int l1 = std::min(l0 + kLevelsPerLaunch, built);
        const int64_t group = 1ll << (2 * (l1 - l0));
        prof_begin(s, st);
        level_build_multi_kernel<<<(unsigned)((lv->cnt[l0] + group - 1) / group), 256, 0, st>>>(nodes, *lv,
                                                                                               l0, l1);
        prof_end(s, st, kStageBuild, 1);
    }
    PBG_CUDA(cudaGetLastError());
    w.sorted_origins_ok = order == kOrderOrigin;
    return PBG_OK;
}

// Pairs per queue buffer: 2^25 (256 MB) unless the scene's parameters set
// another capacity; a batch that overflows it reruns with the triangles split
// into more groups.
constexpr uint32_t kQueueCap = 1u << 25;
constexpr uint32_t kQueueCapMin = 4096;

static uint32_t queue_capacity(const pbg_scene* s) {
    const int32_t q = s->params.rh_queue_pairs;
    return q > 0 ? std::max<uint32_t>((uint32_t)q, kQueueCapMin) : kQueueCap;
}

// Live reach bounds of a nearest-hit batch (words of Work::reach): leaves,
// their parents, then the pair order's buckets.
static bool rh_has_reach(const Levels& lv, bool any) { return !any && lv.nlev > 1; }
static size_t rh_reach_words(const Levels& lv) { return ((size_t)(lv.cnt[0] + lv.cnt[1]) + 3) / 4 * 4; }  // buckets aligned for the scan

// The traversal's buffers, and the words of them that start from zero.
static int rh_workspace(pbg_scene* s, const Levels& lv, bool any, ZeroWords* zero) {
    Work& w = s->work;
    int rc;
    const uint32_t cap = queue_capacity(s);
    if ((rc = ensure(w.queue_a, (size_t)cap * sizeof(Pair))) ||
        (rc = ensure(w.queue_b, (size_t)cap * sizeof(Pair))) ||
        (rc = ensure(w.pair_rank, (size_t)cap * sizeof(uint32_t))) ||
        (rc = ensure(w.leafcnt, (size_t)lv.cnt[0] * sizeof(uint32_t))) ||
        (rc = ensure(w.qcount, 64 * sizeof(uint32_t))))
        return rc;
    zero->add(w.qcount.ptr, 64 * sizeof(uint32_t));
    zero->add((int*)s->err.ptr + kStatusOverflow, sizeof(int));
    const int split = descent_levels(s, lv, any).split;
    if (!(split == 1 && lv.nlev - 1 > split))  // the leaf-pair counting sort runs
        zero->add(w.leafcnt.ptr, (size_t)lv.cnt[0] * sizeof(uint32_t));
    if (rh_has_reach(lv, any)) {
        const size_t bytes = (rh_reach_words(lv) + kOrderBuckets) * sizeof(uint32_t);
        if ((rc = ensure(w.reach, bytes))) return rc;
        zero->add(w.reach.ptr, bytes);
    }
    return PBG_OK;
}

// rh_build has run with the words of rh_workspace zeroed.
template <bool ANY>
static int rh_traverse(pbg_scene* s, const Levels& lv, const float4* so, const float4* sd,
                       unsigned long long* keys, uint32_t* mask, cudaStream_t st, int* moved,
                       const std::function<int(const Publication&)>& finalize) {
    Work& w = s->work;
    int rc;
    const int64_t nleaf = lv.cnt[0];
    const uint32_t cap = queue_capacity(s);
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const bool few = rh_small_batch(nleaf * kLeafRays);
    const int tuned_grid = s->tune.rh_grid[ANY][few];
    const unsigned grid = (unsigned)(sms * (tuned_grid > 0 ? tuned_grid : rh_default_grid(few)));
    const bool stats = s->prof.level >= 2;
    unsigned long long* wc = (unsigned long long*)s->workc.ptr;
    int* status = (int*)s->err.ptr;
    const RayNode* nodes = (const RayNode*)w.nodes.ptr;
    uint32_t* counts = (uint32_t*)w.qcount.ptr;
    constexpr int kNextPair = 2 * kMaxLevels;  // the split tests' next pair
    static_assert(kNextPair < 64, "pair counters");
    int groups = s->rh_groups > 0 ? s->rh_groups : 1;
    const int top = lv.nlev - 1;
    const Descent dsc = descent_levels(s, lv, ANY);
    const int split = dsc.split;
    const int kcl = top - split;  // levels walked by clusters (0: none)
    const float4* tsph = (const float4*)s->spheres.ptr;
    const float4* csph = (const float4*)s->clusters.ptr;
    uint32_t *leaf_reach = nullptr, *parent_reach = nullptr, *order_hist = nullptr;
    if (rh_has_reach(lv, ANY)) {  // live reach bounds, +inf to start (zeroed)
        leaf_reach = (uint32_t*)w.reach.ptr;
        parent_reach = leaf_reach + lv.cnt[0];
        order_hist = leaf_reach + rh_reach_words(lv);
    }
    for (int attempt = 0; attempt < 8; ++attempt) {
        if (attempt > 0) PBG_CUDA(cudaMemsetAsync(status + kStatusOverflow, 0, sizeof(int), st));
        // group boundaries on cluster boundaries
        const int64_t per = ((s->ntri + groups - 1) / groups + kClusterTris - 1) / kClusterTris * kClusterTris;
        for (int g = 0; g < groups; ++g) {
            const int32_t t0 = (int32_t)std::min<int64_t>(s->ntri, g * per),
                          t1 = (int32_t)std::min<int64_t>(s->ntri, (g + 1) * per);
            if (t0 >= t1) break;
            const bool fresh = attempt == 0 && g == 0;  // rh_build zeroed the counters
            if (!fresh) PBG_CUDA(cudaMemsetAsync(counts, 0, 64 * sizeof(uint32_t), st));
            Pair* qa = (Pair*)w.queue_a.ptr;
            Pair* qb = (Pair*)w.queue_b.ptr;
            prof_begin(s, st);
            int nl = 1;  // kernels launched below (scan_counts counts its own)
            // pairs of level l count in counts[l] (clusters: counts[kMaxLevels + l])
            const bool cl = kcl > 0;
            const float4* seed_sph = cl ? csph : tsph;
            const int32_t s0 = cl ? t0 / kClusterTris : t0;
            const int32_t s1 = cl ? (int32_t)((t1 + kClusterTris - 1) / kClusterTris) : t1;
            uint32_t* cnt_of[kMaxLevels];
            for (int l = 0; l < kMaxLevels; ++l) cnt_of[l] = &counts[(cl && l >= split) ? kMaxLevels + l : l];
            // seed level: the lowest with at most kSeedNodes nodes, not below
            // the level where clusters split
            const int ls = dsc.seed;
            const int64_t seed_grid = std::min<int64_t>(
                grid, ((int64_t)(s1 - s0) * lv.cnt[ls] + 255) / 256);
            if (stats)
                rh_seed_kernel<true><<<(unsigned)seed_grid, 256, 0, st>>>(
                    seed_sph, s0, s1, nodes + lv.off[ls], lv.cnt[ls], qa, cnt_of[ls], cap, status, wc);
            else
                rh_seed_kernel<false><<<(unsigned)seed_grid, 256, 0, st>>>(
                    seed_sph, s0, s1, nodes + lv.off[ls], lv.cnt[ls], qa, cnt_of[ls], cap, status,
                    nullptr);
            uint32_t* leafcnt = (uint32_t*)w.leafcnt.ptr;
            uint32_t* rank = (uint32_t*)w.pair_rank.ptr;
            if (!fresh && !(cl && split == 1))  // the leaf-pair counting sort runs
                PBG_CUDA(cudaMemsetAsync(leafcnt, 0, (size_t)nleaf * sizeof(uint32_t), st));
            bool fused = false;
            for (int l = ls; l >= 0; --l) {
                if (cl && l == 1 && split == 1) {  // clusters straight into the leaf tests
                    if (order_hist) {  // nearest: front-to-back pairs, taken in order
                        if (!fresh) PBG_CUDA(cudaMemsetAsync(order_hist, 0, kOrderBuckets * sizeof(uint32_t), st));
                        rh_order_count_kernel<<<grid, 256, 0, st>>>(csph, nodes + lv.off[1], qa, cnt_of[1],
                                                                    cap, order_hist, status);
                        if ((rc = scan_counts(s, order_hist, kOrderBuckets, st))) return rc;
                        rh_order_scatter_kernel<<<grid, 256, 0, st>>>(csph, nodes + lv.off[1], qa,
                                                                      cnt_of[1], cap, order_hist, qb,
                                                                      status);
                        Pair* tq = qa;
                        qa = qb;
                        qb = tq;
                        nl += 2;
                    }
                    const auto kernel = few ? (stats ? rh_split_test_kernel<ANY, true, true> : rh_split_test_kernel<ANY, false, true>)
                                            : (stats ? rh_split_test_kernel<ANY, true, false> : rh_split_test_kernel<ANY, false, false>);
                    kernel<<<(unsigned)(sms * kSplitBlocks), 32 * kSplitWarps, 0, st>>>(
                        tsph, (const TriRec*)s->tris.ptr, t0, t1, nodes + lv.off[1], nodes + lv.off[0], lv.cnt[0], qa,
                        cnt_of[1], cap, counts + kNextPair, so, sd, keys, mask, leaf_reach, parent_reach, status,
                        stats ? wc : nullptr);
                    fused = true;
                    ++nl;
                    break;
                }
                if (cl && l == split) {  // clusters -> triangles, same level
                    if (stats)
                        rh_split_kernel<true><<<grid * 2, 256, 0, st>>>(
                            tsph, t0, t1, nodes + lv.off[l], qa, cnt_of[l], qb, &counts[l], cap,
                            status, wc);
                    else
                        rh_split_kernel<false><<<grid * 2, 256, 0, st>>>(
                            tsph, t0, t1, nodes + lv.off[l], qa, cnt_of[l], qb, &counts[l], cap,
                            status, nullptr);
                    Pair* tq = qa;
                    qa = qb;
                    qb = tq;
                    cnt_of[l] = &counts[l];
                    ++nl;
                }
                if (l == 0) break;
                const float4* sph = (cl && l > split) ? csph : tsph;
                if (stats)
                    rh_expand_kernel<true><<<grid, 256, 0, st>>>(
                        sph, nodes + lv.off[l - 1], lv.cnt[l - 1], qa, cnt_of[l], qb, cnt_of[l - 1],
                        cap, status, wc);
                else
                    rh_expand_kernel<false><<<grid, 256, 0, st>>>(
                        sph, nodes + lv.off[l - 1], lv.cnt[l - 1], qa, cnt_of[l], qb, cnt_of[l - 1],
                        cap, status, nullptr);
                Pair* tq = qa;
                qa = qb;
                qb = tq;
                ++nl;
            }
            // group the leaf pairs by leaf (qa -> qb), then the leaf tests
            if (!fused) {
                rh_leaf_count_kernel<<<grid, 256, 0, st>>>(qa, &counts[0], cap, leafcnt, rank);
                if ((rc = scan_counts(s, leafcnt, nleaf, st))) return rc;
                rh_leaf_scatter_kernel<<<grid, 256, 0, st>>>(qa, &counts[0], cap, leafcnt, rank, qb,
                                                             status);
                if (stats)
                    rh_leaf_sorted_kernel<ANY, true><<<grid * 2, 32 * kLeafWarps, 0, st>>>(
                        (const TriRec*)s->tris.ptr, nodes, qb, &counts[0], cap, so, sd, keys, mask,
                        status, wc);
                else
                    rh_leaf_sorted_kernel<ANY, false><<<grid * 2, 32 * kLeafWarps, 0, st>>>(
                        (const TriRec*)s->tris.ptr, nodes, qb, &counts[0], cap, so, sd, keys, mask,
                        status, nullptr);
                nl += 3;
            }
            prof_end(s, st, kStageTraverse, nl);
            PBG_CUDA(cudaGetLastError());
        }
        // One status read per call: a dropped pair would lose hits.  With
        // *moved, the word after it too: the batch's origins differ from
        // the kept order it was traced in, and the caller traces it again.
        // The finalize kernel runs while the host waits; an attempt that is
        // rerun runs it again.  A small batch's finalize publishes the words
        // itself (a launch less); among a large one's stores the words would
        // reach the host some 15 us later than from a kernel before it.
        Publication pub;
        const int words = moved ? 2 : 1;
        if (few) {
            pub.count = words;
            pub.src = status + kStatusOverflow;
            if ((rc = next_publication(s, &pub.dst, &pub.seq))) return rc;
        } else if ((rc = publish_device_words(s, status + kStatusOverflow, words, &pub.seq, st))) {
            return rc;
        }
        if ((rc = finalize(pub))) return rc;
        int h[2] = {0, 0};
        if ((rc = wait_device_words(s, pub.seq, words, h, st))) return rc;
        if (moved && h[1] != 0) {
            *moved = 1;
            return PBG_OK;
        }
        if (h[0] == 0) return PBG_OK;
        groups *= 4;  // rerun: atomicMax / atomicOr merges make a rerun idempotent
        s->rh_groups = groups;
        s->counters.queue_reruns++;
    }
    set_last_error("rayhierarchy: pair queues overflowed at every triangle grouping");
    return PBG_ERR_INTERNAL;
}

int rh_nearest(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
               int32_t* prim, float* t, float* b1, float* b2, cudaStream_t st) {
    if (n <= 0) return PBG_OK;
    // A nearest-hit batch yields new hit points: the origin order kept for
    // the shadow batches that leave from the previous ones is dropped, so
    // only shadow batches between two nearest-hit batches share a sort.
    s->work.origin_sort_n = -1;
    s->alt.origin_sort_n = -1;
    const int32_t* perm;
    float4 *so, *sd;
    Levels lv;
    Work& w = s->work;
    int rc;
    if ((rc = ensure(w.keys, (size_t)n * 8))) return rc;
    unsigned long long* keys = (unsigned long long*)w.keys.ptr;
    ZeroWords zero;
    zero.add(keys, (size_t)n * 8);
    if ((rc = rh_build(s, o, d, valid, n, &perm, &so, &sd, &lv, kOrderDefault, &zero, st))) return rc;
    const std::function<int(const Publication&)> finalize = [&](const Publication& pub) -> int {
        prof_begin(s, st);
        rh_finalize_nearest<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            (const TriRec*)s->tris.ptr, (const int32_t*)s->tri_pos.ptr, so, sd, perm, keys, n, prim, t, b1,
            b2, pub);
        prof_end(s, st, kStageOther, 1);
        PBG_CUDA(cudaGetLastError());
        return PBG_OK;
    };
    if (s->ntri > 0) return rh_traverse<false>(s, lv, so, sd, keys, nullptr, st, nullptr, finalize);
    return finalize(Publication());
}

int rh_occluded(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
                uint8_t* occ, cudaStream_t st) {
    if (n <= 0) return PBG_OK;
    // Two attempts at most: one in the kept origin order, taken before the
    // comparison's answer, and, when the origins moved, one in a fresh order
    // (the kept order is dropped, so that attempt cannot speculate).
    for (int attempt = 0; attempt < 2; ++attempt) {
        const int32_t* perm;
        float4 *so, *sd;
        Levels lv;
        Work& w = s->work;
        const size_t mask_bytes = (size_t)((n + kLeafRays - 1) / kLeafRays) * 4;
        int rc;
        if ((rc = ensure(w.leafmask, mask_bytes))) return rc;
        uint32_t* mask = (uint32_t*)w.leafmask.ptr;
        ZeroWords zero;
        zero.add(mask, mask_bytes);
        if ((rc = rh_build(s, o, d, valid, n, &perm, &so, &sd, &lv, kOrderOrigin, &zero, st))) return rc;
        const bool speculative = w.origin_speculative;
        const std::function<int(const Publication&)> finalize = [&](const Publication& pub) -> int {
            prof_begin(s, st);
            rh_finalize_occluded<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(perm, mask, n, occ, pub);
            prof_end(s, st, kStageOther, 1);
            PBG_CUDA(cudaGetLastError());
            return PBG_OK;
        };
        int moved = 0;
        if (s->ntri > 0) {
            // the finalize runs behind the status publication; a moved
            // batch's answers are overwritten by the next attempt's
            rc = rh_traverse<true>(s, lv, so, sd, nullptr, mask, st, speculative ? &moved : nullptr, finalize);
            if (rc) return rc;
        } else {
            if ((rc = finalize(Publication()))) return rc;
            if (speculative &&
                (rc = read_device_words(s, (const int*)s->err.ptr + kStatusOriginMoved, 1, &moved, st)))
                return rc;
        }
        if (moved) {
            w.origin_sort_n = -1;
            w.origin_reused = w.origin_speculative = false;
            s->counters.origin_reruns++;
            continue;
        }
        if (speculative) s->counters.origin_reuses++;
        return PBG_OK;
    }
    set_last_error("rayhierarchy: the origin order changed under a fresh sort");
    return PBG_ERR_INTERNAL;
}

}  // namespace pbg
