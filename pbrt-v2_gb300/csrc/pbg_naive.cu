// pbg_naive.cu -- Accelerator "naive": every ray against every triangle that
// it can hit.
//
// Replaces the fork's all-pairs OpenCL kernels (bin/cl/naive.cl:4-231, one
// thread per triangle looping over rays, racing on tHit; bin/cl/naive2.cl,
// one thread per ray) and their host side (accelerators/naive.cpp:204-437).
// Results follow pbrt's CPU test exactly instead of those kernels' widened
// epsilons (naive.cl:2, :32, :38).
//
// The records are kept along a Hilbert curve of their centroids, in groups of
// 32 with a box each, and a warp of 32 rays skips the pairs that cannot hit.
// A pair is skipped only where pbrt's float test provably rejects it, so the
// answer stays that of the loop over all triangles; no tree is involved.
//
// The proof (u = 2^-24; d direction, v = o - p1, N a member's unit normal, E
// its longest edge from p1, phi the angle between its edges).  Every triple
// product that the test forms is within 5.3 u of the product of its three
// vectors' lengths of the real one: Cross() rounds each component once
// (1.01 u of |ab| + |cd|, whose three components have a norm of at most
// 1.155 |a| |b|), Dot() adds 3 roundings, v another.  The groups hold only
// triangles with sin(phi) >= 2^-4 (the others are tested by every ray).
//   A. |d.N| >= 2^-4 |d|: the divisor is within 8.1e-5 of itself, each
//      barycentric within 8.1e-5 (1 + |v| / edge), and t |d| within 1.7e-4
//      (|v| + E).  A hit that the test accepts therefore lies, at its own
//      t, within 4.1e-4 (|v| + E) of the triangle: the ray passes through
//      the group's box grown by 2^-10 (|v| + E) at a t in [mint, maxt].
//   B. |d.N| < 2^-4 |d|: b1 and b2 in [0, 1] bound the in-plane part of v x d
//      by |d| (|d.N| / |d|) 2 E + 1e-5 |v| |d|, and that part is at least
//      |v.N| |d| (1 - 2^-8)^(1/2) - |d.N| |v|; so |v.N| <= 0.0628 (|v| + 2 E).
// So a member can be hit by a ray that misses the grown box only if the ray
// runs nearly within the member's plane.  A warp bounds its rays by one cone
// and one origin ball: each lane looks at one member of a group, and the few
// that some ray of the warp may see edge on (2 to 3 % of them) are tested
// whatever the box says; the others are tested by the rays that meet the box.
// A warp whose rays do not fit a cone of 20 degrees tests everything, as do
// rays of extreme size; triangles of extreme size (edges below 2^-30 or
// coordinates above 2^30, where underflow or overflow would enter the bounds)
// are among those that every ray tests.
//
// Work: one thread per ray, the group range split across gridDim.y so that
// small batches still fill the SMs.  A group's records are staged in shared
// memory by the warp and tested ray per lane, or triangle per lane for a few
// rays.  With one split the thread writes its hit directly; with several, the
// splits merge through a 64-bit atomicMax on (t, index) keys and a finalize
// pass recomputes b1/b2 of the winner with the exact test.
//
// Bound by instruction issue.  65,536 camera rays and their shadow rays
// against the 4,034 triangles of a sphere over a quad: 697 us with
// every pair tested, 170 us with groups skipped.
#include <algorithm>

#include "pbg_count.cuh"
#include "pbg_curve.cuh"
#include "pbg_internal.h"
#include "pbg_walk.cuh"

namespace pbg {

int radix_sort_pairs(pbg_scene* s, uint32_t* keys, int32_t* vals, uint32_t* keys_tmp, int32_t* vals_tmp,
                     uint32_t* hist, int64_t n, int bits, uint32_t** keys_out, int32_t** vals_out,
                     cudaStream_t st);
size_t radix_hist_words(int64_t n);

constexpr int kNaiveThreads = 128;
constexpr int kNaiveGroup = 32;       // records per group: one per lane
constexpr int kNaiveKeyBits = 24;     // Hilbert index of the centroid, 8 bits per axis
// A kept group is tested triangle per lane for fewer kept rays than this: a
// ray's turn costs about 50 instructions, the loop over the 32 records 960.
constexpr int kNaiveDense = 18;
constexpr float kNaiveGrow = 0x1p-10f;   // A: 4.1e-4 needed
constexpr float kNaiveTau = 0x1p-4f;
constexpr float kNaiveKappa = 0.064f;    // B: 0.0628 needed
constexpr float kNaiveCone = 0.94f;      // least cosine of a warp's direction cone

struct __align__(16) NaiveGroup {
    float4 c;  // box centre
    float4 h;  // half extents with the part of their growth that no ray changes
};

// ---------------------------------------------------------------- build

__device__ __forceinline__ int ordered_int(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// Whether a triangle may be skipped (the file header's conditions).
__device__ bool skippable(const float* v) {
    double e1[3], e2[3], l1 = 0.0, l2 = 0.0;
    for (int k = 0; k < 9; ++k)
        if (!(fabsf(v[k]) <= 0x1p30f)) return false;
    for (int k = 0; k < 3; ++k) {
        e1[k] = (double)__fsub_rn(v[3 + k], v[k]);
        e2[k] = (double)__fsub_rn(v[6 + k], v[k]);
        l1 += e1[k] * e1[k];
        l2 += e2[k] * e2[k];
    }
    if (!(l1 >= 0x1p-60) || !(l2 >= 0x1p-60)) return false;
    const double cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2],
                 cz = e1[0] * e2[1] - e1[1] * e2[0];
    return cx * cx + cy * cy + cz * cz >= 0x1.001p-8 * l1 * l2;
}

// words: [0-2] least centroid, [3-5] greatest (ordered ints), [6] triangles
// that every ray tests.
__global__ void naive_init_kernel(int* __restrict__ words) {
    if (threadIdx.x < 8) words[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : threadIdx.x < 6 ? (int)0x80000000 : 0;
}

__device__ __forceinline__ float centroid(const float* v, int a) { return (v[a] + v[3 + a] + v[6 + a]) * (1.f / 3.f); }

__global__ void __launch_bounds__(256)
    naive_prep_kernel(const float* __restrict__ tri9, int64_t n, uint8_t* __restrict__ skip, int* __restrict__ words) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const float* v = tri9 + 9 * i;
    const bool in = i < n, ok = in && skippable(v);
    if (in) skip[i] = ok ? 1 : 0;
    const int c = __syncthreads_count(in && !ok);
    if (threadIdx.x == 0 && c) atomicAdd(&words[6], c);
    for (int a = 0; a < 3; ++a) {
        float lo = ok ? centroid(v, a) : INFINITY, hi = ok ? lo : -INFINITY;
        for (int off = 16; off; off >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&words[a], ordered_int(lo));
            atomicMax(&words[3 + a], ordered_int(hi));
        }
    }
}

// Sort keys: 0 for the triangles that every ray tests, else 1 + the centroid's
// position along a Hilbert curve of cubic cells (Morton order left groups
// twice as large).
__global__ void __launch_bounds__(256)
    naive_key_kernel(const float* __restrict__ tri9, int64_t n, const uint8_t* __restrict__ skip,
                     const int* __restrict__ words, uint32_t* __restrict__ keys, int32_t* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vals[i] = (int32_t)i;
    if (!skip[i]) {
        keys[i] = 0u;
        return;
    }
    float ext = 0.f;
    for (int a = 0; a < 3; ++a) ext = fmaxf(ext, from_ordered(words[3 + a]) - from_ordered(words[a]));
    uint32_t q[3];
    for (int a = 0; a < 3; ++a) {
        const float x = ext > 0.f ? (centroid(tri9 + 9 * i, a) - from_ordered(words[a])) / ext * 256.f : 0.f;
        q[a] = (uint32_t)fminf(fmaxf(x, 0.f), 255.f);
    }
    hilbert3(q, 8);
    keys[i] = min(((spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2])) + 1u, (1u << kNaiveKeyBits) - 2u);
}

// One warp per group, one lane per member (order[first + lane]): the group's
// box, and each member's unit normal and longest edge.
__global__ void __launch_bounds__(256)
    naive_group_kernel(const float* __restrict__ tri9, const int32_t* __restrict__ order, const int* __restrict__ words,
                       int64_t n, NaiveGroup* __restrict__ groups, float4* __restrict__ normals) {
    const int lane = threadIdx.x & 31;
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t first = (int64_t)words[6] + g * kNaiveGroup;
    if (first >= n) return;
    const int64_t i = first + lane;
    const float* v = tri9 + 9 * (int64_t)order[i < n ? i : first];  // a lane past the end repeats the first member
    float lo[3], hi[3];
    double e1[3], e2[3], l1 = 0.0, l2 = 0.0;
    for (int a = 0; a < 3; ++a) {
        lo[a] = fminf(v[a], fminf(v[3 + a], v[6 + a]));
        hi[a] = fmaxf(v[a], fmaxf(v[3 + a], v[6 + a]));
        e1[a] = (double)v[3 + a] - (double)v[a];
        e2[a] = (double)v[6 + a] - (double)v[a];
        l1 += e1[a] * e1[a];
        l2 += e2[a] * e2[a];
    }
    const double nx = e1[1] * e2[2] - e1[2] * e2[1], ny = e1[2] * e2[0] - e1[0] * e2[2],
                 nz = e1[0] * e2[1] - e1[1] * e2[0];
    const double inv = 1.0 / sqrt(nx * nx + ny * ny + nz * nz);
    float e = (float)(sqrt(fmax(l1, l2)) * (1.0 + 0x1p-20));
    if (i < n) normals[i] = make_float4((float)(nx * inv), (float)(ny * inv), (float)(nz * inv), e);
    for (int off = 16; off; off >>= 1) {
        e = fmaxf(e, __shfl_xor_sync(0xffffffffu, e, off));
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    if (lane != 0) return;
    float c[3], h[3], mag = 0.f;
    for (int a = 0; a < 3; ++a) {
        c[a] = 0.5f * lo[a] + 0.5f * hi[a];
        h[a] = fmaxf(hi[a] - c[a], c[a] - lo[a]);
        mag = fmaxf(mag, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
    }
    // the farthest member corner from the centre, and the growth that does
    // not depend on the ray (2^-20 of the coordinates for the edges' and the
    // centre's own rounding)
    const float r = sqrtf(h[0] * h[0] + h[1] * h[1] + h[2] * h[2]) * (1.f + 0x1p-18f) + 0x1p-20f * mag;
    const float grow = kNaiveGrow * 1.01f * (r + e) + 0x1p-20f * mag;
    groups[g] = NaiveGroup{make_float4(c[0], c[1], c[2], 0.f), make_float4(h[0] + grow, h[1] + grow, h[2] + grow, 0.f)};
}

int naive_build(pbg_scene* s, DeviceBuffer& order) {
    const int64_t n = s->ntri;
    cudaStream_t st = s->stream;
    s->unculled = 0;
    if (n <= 0) return PBG_OK;
    DeviceBuffer skip, keys, keys_tmp, vals, hist, words;
    struct Guard {
        DeviceBuffer* b[6];
        ~Guard() {
            for (DeviceBuffer* x : b) release(*x);
        }
    } guard{{&skip, &keys, &keys_tmp, &vals, &hist, &words}};
    int rc;
    if ((rc = ensure(skip, (size_t)n)) || (rc = ensure(keys, (size_t)n * 4)) || (rc = ensure(keys_tmp, (size_t)n * 4)) ||
        (rc = ensure(vals, (size_t)n * 4)) || (rc = ensure(order, (size_t)n * 4)) ||
        (rc = ensure(hist, radix_hist_words(n) * 4)) || (rc = ensure(words, 32)) ||
        (rc = ensure(s->naive_groups, (size_t)((n + kNaiveGroup - 1) / kNaiveGroup) * sizeof(NaiveGroup))) ||
        (rc = ensure(s->naive_normals, (size_t)n * sizeof(float4))))
        return rc;
    const float* tri9 = (const float*)s->tri9.ptr;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    naive_init_kernel<<<1, 32, 0, st>>>((int*)words.ptr);
    naive_prep_kernel<<<blocks, 256, 0, st>>>(tri9, n, (uint8_t*)skip.ptr, (int*)words.ptr);
    // an odd number of passes ends in the second pair of buffers
    naive_key_kernel<<<blocks, 256, 0, st>>>(tri9, n, (const uint8_t*)skip.ptr, (const int*)words.ptr, (uint32_t*)keys.ptr,
                                             (int32_t*)vals.ptr);
    PBG_CUDA(cudaGetLastError());
    uint32_t* ks;
    int32_t* vs;
    if ((rc = radix_sort_pairs(s, (uint32_t*)keys.ptr, (int32_t*)vals.ptr, (uint32_t*)keys_tmp.ptr, (int32_t*)order.ptr,
                               (uint32_t*)hist.ptr, n, kNaiveKeyBits, &ks, &vs, st)))
        return rc;
    if (vs != (int32_t*)order.ptr) PBG_CUDA(cudaMemcpyAsync(order.ptr, vs, (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
    naive_group_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(tri9, (const int32_t*)order.ptr, (const int*)words.ptr, n,
                                                                  (NaiveGroup*)s->naive_groups.ptr,
                                                                  (float4*)s->naive_normals.ptr);
    PBG_CUDA(cudaGetLastError());
    s->counters.kernel_launches += 4;
    int h[8];
    PBG_CUDA(cudaMemcpyAsync(h, words.ptr, 32, cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaStreamSynchronize(st));
    s->unculled = h[6];
    return PBG_OK;
}

// -------------------------------------------------------------- traverse

// A bound over the warp's live rays: unit directions within the cone (axis,
// cos, sin), origins within the ball (o, r).
struct Bundle {
    float ox, oy, oz, r, dx, dy, dz, cs, sn;
};

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// False when the live rays have no bound worth using.
__device__ __forceinline__ bool make_bundle(bool live, float4 o, float4 d, float nd, Bundle* b) {
    const bool plain = nd >= 0x1p-30f && nd <= 0x1p30f && fabsf(o.x) + fabsf(o.y) + fabsf(o.z) <= 0x1p30f;
    if (__any_sync(0xffffffffu, live && !plain)) return false;
    const float il = live ? rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z) : 0.f;
    const float ux = d.x * il, uy = d.y * il, uz = d.z * il;
    float sx = live ? ux : 0.f, sy = live ? uy : 0.f, sz = live ? uz : 0.f;
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sz += __shfl_xor_sync(0xffffffffu, sz, off);
    }
    const float sl = rsqrtf(sx * sx + sy * sy + sz * sz);
    b->dx = sx * sl;
    b->dy = sy * sl;
    b->dz = sz * sl;
    // the units' and the axis's own rounding: 2^-18
    b->cs = -warp_max(live ? -(ux * b->dx + uy * b->dy + uz * b->dz) : -1.f) - 0x1p-18f;
    if (!(b->cs > kNaiveCone)) return false;
    b->sn = sqrtf(fmaxf(0.f, 1.f - b->cs * b->cs)) + 0x1p-18f;
    b->ox = 0.5f * (warp_max(live ? o.x : -INFINITY) - warp_max(live ? -o.x : -INFINITY));
    b->oy = 0.5f * (warp_max(live ? o.y : -INFINITY) - warp_max(live ? -o.y : -INFINITY));
    b->oz = 0.5f * (warp_max(live ? o.z : -INFINITY) - warp_max(live ? -o.z : -INFINITY));
    const float x = o.x - b->ox, y = o.y - b->oy, z = o.z - b->oz;
    b->r = warp_max(live ? sqrtf(x * x + y * y + z * z) : 0.f) * (1.f + 0x1p-18f) +
           0x1p-20f * (fabsf(b->ox) + fabsf(b->oy) + fabsf(b->oz));
    return true;
}

// Whether some ray of the bundle may run nearly within the plane of the
// triangle with unit normal and longest edge ne, first vertex p (the file
// header's cases A and B, each with 2^-16 to spare for the arithmetic here).
__device__ __forceinline__ bool edge_on(const Bundle& b, float4 ne, float4 p) {
    const float da = fabsf(b.dx * ne.x + b.dy * ne.y + b.dz * ne.z);
    if (da * b.cs - b.sn >= kNaiveTau + 0x1p-16f) return false;  // A
    const float vx = b.ox - p.x, vy = b.oy - p.y, vz = b.oz - p.z;
    const float vl = sqrtf(vx * vx + vy * vy + vz * vz);
    const float va = fabsf(vx * ne.x + vy * ne.y + vz * ne.z);
    return !(va - b.r > (kNaiveKappa + 0x1p-16f) * (vl + b.r + 2.f * ne.w));  // not B
}

// STATS: the counting variant (profiling level 2) adds each thread's box
// tests, filter tests, second-stage filter passes, exact tests and exact
// hits to wcount.
template <bool ANY, bool STATS>
__global__ void __launch_bounds__(kNaiveThreads)
    naive_kernel(const TriRec* __restrict__ tris, const NaiveGroup* __restrict__ groups,
                 const float4* __restrict__ normals, int32_t ntri, int32_t unculled, int32_t ngroups, int32_t per_split,
                 const float4* __restrict__ ro, const float4* __restrict__ rd,
                 const uint8_t* __restrict__ valid, int64_t n, int32_t* __restrict__ prim_out,
                 float* __restrict__ t_out, float* __restrict__ b1_out,
                 float* __restrict__ b2_out, unsigned long long* __restrict__ keys,
                 uint8_t* __restrict__ occ, unsigned long long* wcount) {
    __shared__ TriRec stage[kNaiveThreads / 32][kNaiveGroup];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    TriRec* rec = stage[threadIdx.x >> 5];
    const int64_t ray = (int64_t)blockIdx.x * kNaiveThreads + threadIdx.x;
    const bool split = gridDim.y > 1;
    const bool active = ray < n && (valid == nullptr || valid[ray] != 0);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
    if (active) {
        o = ro[ray];
        d = rd[ray];
    }
    const float nd = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    const float ix = safe_inv(d.x), iy = safe_inv(d.y), iz = safe_inv(d.z);
    WalkHit h{d.w, 0.f, 0.f, -1};
    bool done = !active;
    WorkCount wc;
    Bundle bd;
    const bool bundle = make_bundle(active, o, d, nd, &bd);
    const bool idle = __all_sync(full, done);  // no valid ray

    auto test = [&](const TriRec& tr) {
        if (STATS) wc.filt++;
        if (!pbg_filter<true>(tr, o, d, nd, h.t, STATS ? &wc.filt2 : nullptr)) return;
        float tt, u1, u2;
        if (STATS) wc.exact++;
        if (!pbg_exact_rec(tr, o, d, h.t, &tt, &u1, &u2)) return;
        if (STATS) wc.hit++;
        const int32_t id = __float_as_int(tr.c.w);
        if (ANY) {
            h.prim = id;
            done = true;
        } else if (tt < h.t || id > h.prim) {
            h = WalkHit{tt, u1, u2, id};
        }
    };
    // this warp's next 32 records, one per lane, in shared memory
    auto load = [&](int32_t first, int32_t cnt) {
        __syncwarp();
        if (lane < cnt) rec[lane] = tris[first + lane];
        __syncwarp();
    };
    auto test_all = [&](int32_t cnt) {
        if (cnt == kNaiveGroup) {
#pragma unroll 4
            for (int32_t j = 0; j < kNaiveGroup; ++j)
                if (!done) test(rec[j]);
        } else {
            for (int32_t j = 0; j < cnt; ++j)
                if (!done) test(rec[j]);
        }
    };

    // the triangles that every ray tests, shared out over the splits; a warp
    // leaves once its rays are occluded, or if none of them is valid
    const int32_t u0 = (int32_t)((int64_t)unculled * blockIdx.y / gridDim.y);
    const int32_t u1 = (int32_t)((int64_t)unculled * (blockIdx.y + 1) / gridDim.y);
    for (int32_t j = u0; j < u1; j += kNaiveGroup) {
        if (ANY ? __all_sync(full, done) : idle) break;
        load(j, min(kNaiveGroup, u1 - j));
        test_all(min(kNaiveGroup, u1 - j));
    }
    const int32_t g0 = min((int32_t)blockIdx.y * per_split, ngroups), g1 = min(g0 + per_split, ngroups);
    for (int32_t g = g0; g < g1; ++g) {
        if (ANY ? __all_sync(full, done) : idle) break;
        const int32_t first = unculled + g * kNaiveGroup;
        const int32_t cnt = min(kNaiveGroup, ntri - first);
        unsigned meet = full, side = 0;  // lanes whose rays test every member; members that the others test too
        if (bundle) {
            const NaiveGroup gr = groups[g];
            const float vx = gr.c.x - o.x, vy = gr.c.y - o.y, vz = gr.c.z - o.z;
            const float v2 = vx * vx + vy * vy + vz * vz;
            // |v| rounded up (0 and overflow: NaN, which keeps the group)
            const float vl = v2 * rsqrtf(v2) * (1.f + 0x1p-18f);
            const float tx = vx * ix, ty = vy * iy, tz = vz * iz;
            const float wx = fmaf(kNaiveGrow, vl, gr.h.x) * fabsf(ix), wy = fmaf(kNaiveGrow, vl, gr.h.y) * fabsf(iy),
                        wz = fmaf(kNaiveGrow, vl, gr.h.z) * fabsf(iz);
            const float tn = fmax3(tx - wx, ty - wy, fmaxf(tz - wz, o.w));
            const float tf = fmin3(tx + wx, ty + wy, fminf(tz + wz, h.t));
            if (STATS && !done) wc.node++;
            meet = __ballot_sync(full, !done && !(tn > tf));
            if (__popc(meet) < kNaiveDense)
                side = __ballot_sync(full, lane < cnt && edge_on(bd, normals[first + lane], tris[first + lane].a));
            if (meet == 0 && side == 0) continue;
        }
        if (STATS && lane == 0) wc.leaf++;
        load(first, cnt);
        if (__popc(meet) >= kNaiveDense) {  // ray per lane
            test_all(cnt);
            continue;
        }
        for (unsigned m = meet; m; m &= m - 1) {  // triangle per lane, those rays in turn
            const int i = __ffs(m) - 1;
            const float4 oi = make_float4(__shfl_sync(full, o.x, i), __shfl_sync(full, o.y, i),
                                          __shfl_sync(full, o.z, i), __shfl_sync(full, o.w, i));
            const float4 di = make_float4(__shfl_sync(full, d.x, i), __shfl_sync(full, d.y, i),
                                          __shfl_sync(full, d.z, i), 0.f);
            const float ni = __shfl_sync(full, nd, i), mi = __shfl_sync(full, h.t, i);
            float tt = 0.f, b1 = 0.f, b2 = 0.f;
            bool hit = false;
            if (lane < cnt) {
                const TriRec own = rec[lane];
                if (STATS) wc.filt++;
                if (pbg_filter<true>(own, oi, di, ni, mi, STATS ? &wc.filt2 : nullptr)) {
                    if (STATS) wc.exact++;
                    hit = pbg_exact_rec(own, oi, di, mi, &tt, &b1, &b2);
                    if (STATS && hit) wc.hit++;
                }
            }
            for (unsigned hm = __ballot_sync(full, hit); hm; hm &= hm - 1) {  // seldom more than one
                const int k = __ffs(hm) - 1;
                const float kt = __shfl_sync(full, tt, k), k1 = __shfl_sync(full, b1, k), k2 = __shfl_sync(full, b2, k);
                const int32_t id = __float_as_int(rec[k].c.w);
                if (lane == i) {
                    if (ANY) {
                        h.prim = id;
                        done = true;
                    } else if (kt < h.t || (!(kt > h.t) && id > h.prim)) {
                        h = WalkHit{kt, k1, k2, id};
                    }
                }
            }
        }
        for (; side; side &= side - 1)
            if (!done && !(meet >> lane & 1u)) test(rec[__ffs(side) - 1]);
    }
    if (STATS) wc.flush(wcount);
    if (ray >= n) return;
    if (ANY) {
        if (split) {
            if (h.prim >= 0) occ[ray] = 1;
        } else {
            occ[ray] = h.prim >= 0 ? 1 : 0;
        }
        return;
    }
    if (split) {
        if (h.prim >= 0) atomicMax(&keys[ray], hit_key(h.t, h.prim));
        return;
    }
    const bool hit = h.prim >= 0;
    prim_out[ray] = h.prim;
    t_out[ray] = hit ? h.t : 0.f;
    b1_out[ray] = hit ? h.b1 : 0.f;
    b2_out[ray] = hit ? h.b2 : 0.f;
}

// Turns merged (t, index) keys into hits; b1/b2 (and t) of the winner come
// from the exact test again, which is deterministic.  pos maps an original
// triangle index to its record (NULL = identity).
__global__ void finalize_keys_kernel(const TriRec* __restrict__ tris, const int32_t* __restrict__ pos,
                                     const float4* __restrict__ ro, const float4* __restrict__ rd,
                                     const unsigned long long* __restrict__ keys, int64_t n,
                                     int32_t* prim, float* t, float* b1, float* b2) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = keys[i];
    int32_t p = -1;
    float tt = 0.f, u1 = 0.f, u2 = 0.f;
    if (k != 0ull) {
        p = key_prim(k);
        const TriRec tr = tris[pos ? pos[p] : p];
        const float4 o = ro[i], d = rd[i];
        if (!pbg_exact_rec(tr, o, d, d.w, &tt, &u1, &u2)) {
            p = -1;  // unreachable: the key came from this same test
            tt = u1 = u2 = 0.f;
        }
    }
    prim[i] = p;
    t[i] = tt;
    b1[i] = u1;
    b2[i] = u2;
}

int finalize_keys(pbg_scene* s, const int32_t* pos, const float4* o, const float4* d,
                  const unsigned long long* keys, int64_t n, int32_t* prim, float* t, float* b1,
                  float* b2, cudaStream_t st) {
    if (n <= 0) return PBG_OK;
    const int threads = 256;
    prof_begin(s, st);
    finalize_keys_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, st>>>(
        (const TriRec*)s->tris.ptr, pos, o, d, keys, n, prim, t, b1, b2);
    prof_end(s, st, kStageOther, 1);
    PBG_CUDA(cudaGetLastError());
    return PBG_OK;
}

// The group range is cut so that about tune.naive_ctas CTAs per SM (16 unless
// tuned: 181 / 170 / 181 us for 8 / 16 / 32 at the sizes above, 256-thread
// CTAs 191 / 210 / 240) run; a split may be one group, since in a small batch
// the warps run their groups one after another on an idle chip (1,200 rays and
// as many shadow rays on 4,000 triangles: 72 us with at least four, 48 so; all
// pairs: 62).
static void naive_launch_shape(pbg_scene* s, int64_t n, int32_t* ngroups, int32_t* per_split, unsigned* splits) {
    const int64_t ray_ctas = (n + kNaiveThreads - 1) / kNaiveThreads;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const int64_t per_sm = s->tune.naive_ctas > 0 ? s->tune.naive_ctas : 16;
    const int64_t ng = (s->ntri - s->unculled + kNaiveGroup - 1) / kNaiveGroup;
    // the triangles that every ray tests count as groups of their own here
    const int64_t units = ng + (s->unculled + kNaiveGroup - 1) / kNaiveGroup;
    int64_t want = (per_sm * (int64_t)sms + ray_ctas - 1) / ray_ctas;
    want = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, units), 65535));
    *ngroups = (int32_t)ng;
    *per_split = (int32_t)((ng + want - 1) / want);
    *splits = (unsigned)want;
}

template <bool ANY>
static int naive_launch(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n, int32_t* prim,
                        float* t, float* b1, float* b2, uint8_t* occ, cudaStream_t st) {
    if (n <= 0) return PBG_OK;
    int32_t ngroups, per;
    unsigned splits;
    naive_launch_shape(s, n, &ngroups, &per, &splits);
    unsigned long long* keys = nullptr;
    if (splits > 1 && ANY) PBG_CUDA(cudaMemsetAsync(occ, 0, (size_t)n, st));
    if (splits > 1 && !ANY) {
        const int rc = ensure(s->work.keys, (size_t)n * sizeof(unsigned long long));
        if (rc) return rc;
        keys = (unsigned long long*)s->work.keys.ptr;
        PBG_CUDA(cudaMemsetAsync(keys, 0, (size_t)n * sizeof(unsigned long long), st));
    }
    const bool stats = s->prof.level >= 2;
    auto kern = stats ? naive_kernel<ANY, true> : naive_kernel<ANY, false>;
    prof_begin(s, st);
    kern<<<dim3((unsigned)((n + kNaiveThreads - 1) / kNaiveThreads), splits), kNaiveThreads, 0, st>>>(
        (const TriRec*)s->tris.ptr, (const NaiveGroup*)s->naive_groups.ptr, (const float4*)s->naive_normals.ptr,
        (int32_t)s->ntri, s->unculled, ngroups, per, o, d, valid, n, prim, t, b1, b2, keys, occ, stats ? (unsigned long long*)s->workc.ptr : nullptr);
    prof_end(s, st, kStageTraverse, 1);
    PBG_CUDA(cudaGetLastError());
    if (splits > 1 && !ANY)
        return finalize_keys(s, (const int32_t*)s->tri_pos.ptr, o, d, keys, n, prim, t, b1, b2, st);
    return PBG_OK;
}

int naive_nearest(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
                  int32_t* prim, float* t, float* b1, float* b2, cudaStream_t st) {
    return naive_launch<false>(s, o, d, valid, n, prim, t, b1, b2, nullptr, st);
}

int naive_occluded(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
                   uint8_t* occ, cudaStream_t st) {
    return naive_launch<true>(s, o, d, valid, n, nullptr, nullptr, nullptr, nullptr, occ, st);
}

}  // namespace pbg
