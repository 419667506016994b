// pbg_render.cu -- the breadth-first renderer as a device wavefront.
//
// Reference: renderers/breadth-first.cpp:18-228 generates every camera ray
// of a task tile, calls the batch Li of the surface integrator, which shades
// on the host and sends shadow rays (core/integrator.cpp:73-455) and bounce
// rays (integrators/path.cpp:43-157) back as batches; rays that die keep
// their slot.  Here the whole image is one batch and every stage runs on the
// device:
//
//   raygen     camera rays from the caller's RasterToCamera / CameraToWorld
//              (cameras/perspective.cpp GenerateRayDifferential), stratified
//              image samples (samplers/stratified.cpp), scanline order with
//              spp consecutive samples (the breadth-first ray image);
//   trace      the scene's accelerator (pbg_*_device) on the live queue;
//   shade      Lambertian BSDF (core/reflection.cpp:165), light sampling
//              (lights/point.cpp; lights/diffuse.cpp over scene triangles as
//              ShapeSet samples them, core/light.cpp:137-165; a
//              parallelogram emitter), the batch integrators' EstimateDirect
//              (core/integrator.cpp:212-298 for path, :358-455 for
//              directlighting, each with its own operation order), emission
//              at camera hits on emitting triangles, one shadow slot per
//              light sample and one bounce slot per path;
//   append     shade puts its shadow and bounce rays straight into the next
//              queues: ballots give ranks inside a block, one atomic per block
//              its place (stream renders, whose draws follow the queue's
//              order, flag slots and compact them in order instead);
//   resolve    unoccluded shadow contributions added per sample in light
//              sample order (deterministic, no float atomics);
//   film       per pixel, samples in order, through XYZ as ImageFilm does
//              (film/image.cpp AddSample / WriteImage), box filter; samples
//              whose radiance breadthFirst::Li would reject (NaN, negative or
//              infinite luminance) count as black.
//
// Random numbers: by default a counter-based hash of (seed, sample,
// dimension), identical on every run and in the oracle's restatement.  With
// a sample stream (pbg_render_stream) the values are the reference's own:
// the caller passes one task's samples as pbrt's StratifiedSampler drew them
// and the continuation of the task's RNG, which the renderer consumes in
// the order the batch integrators do -- path tracing below bounce 3 reads
// the sample arrays (integrators/path.cpp:31-38), from bounce 3 on
// UniformSampleOneLight draws 7 values for every ray of the task, then each
// ray that hit draws its BSDF sample (3) and, after bounce 3, its Russian
// roulette value (1), in ray order (core/integrator.cpp:142-165,
// integrators/path.cpp:104-124).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pbg_dg.cuh"
#include "pbg_internal.h"
#include "pbg_learn.h"
#include "pbg_tma.cuh"

namespace pbg {

constexpr float kInvPi = 0.31830988618379067154f;

// splitmix64 finalizer (a published 64-bit mixing function)
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Uniform float in [0, 1) for (seed, sample, dim).
__device__ __forceinline__ float rnd(uint64_t seed, uint64_t sample, uint32_t dim) {
    const uint64_t h = mix64(seed ^ mix64(sample * 0x100000001B3ull + dim));
    return (float)(h >> 40) * 0x1p-24f;
}

// Sample dimensions: 0-1 image, then 16 per bounce: light samples from 0,
// Russian roulette at 13, BSDF sample at 14-15.  The light-sample
// components of triangle emitters and the light choice of the path
// integrator use a second family from 512.
__device__ __forceinline__ uint32_t dim_of(int bounce, int k) { return 2u + 16u * (uint32_t)bounce + (uint32_t)k; }
__device__ __forceinline__ uint32_t dim_extra(int bounce, int k) { return 512u + 16u * (uint32_t)bounce + (uint32_t)k; }
constexpr int kDimRR = 13, kDimBsdf = 14;

// sin and cos in float from the Cephes single-precision polynomials
// (S. Moshier, Cephes Math Library, sinf.c/cosf.c coefficients) after a
// two-constant Cody-Waite reduction by pi/2, every operation correctly
// rounded and unfused, so the oracle's C restatement gives identical bits.
__device__ __forceinline__ void own_sincos(float a, float* s, float* c) {
    const float jf = rintf(__fmul_rn(a, 0.636619772367581343f));
    const int j = (int)jf;
    const float r = __fsub_rn(__fsub_rn(a, __fmul_rn(jf, 1.5703125f)), __fmul_rn(jf, 4.83826794897e-4f));
    const float z = __fmul_rn(r, r);
    const float sp = __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(__fmul_rn(__fadd_rn(__fmul_rn(-1.9515295891e-4f, z),
                                                                                    8.3321608736e-3f), z),
                                                               1.6666654611e-1f), z), r), r);
    const float cp = __fadd_rn(__fsub_rn(__fmul_rn(__fmul_rn(__fadd_rn(__fmul_rn(__fsub_rn(__fmul_rn(2.443315711809948e-5f, z),
                                                                                              1.388731625493765e-3f), z),
                                                                          4.166664568298827e-2f), z), z),
                                         __fmul_rn(0.5f, z)), 1.f);
    switch (j & 3) {
        case 0: *s = sp; *c = cp; break;
        case 1: *s = cp; *c = -sp; break;
        case 2: *s = -sp; *c = -cp; break;
        default: *s = -cp; *c = sp; break;
    }
}

struct DevLight {
    int type, nsamples;
    float pos[3], I[3];
    float q0[3], e1[3], e3[3], n[3], area, L[3];
    int first, ntri;  // triangle emitter: scene triangles [first, first + ntri)
    int tab;          // ... its areas, CDF and total area in the light table
};

struct RenderConst {
    float r2c[16], c2w[16];
    int xres, yres, spp_x, spp_y, spp, jitter, max_depth, integrator;
    uint64_t seed;
    float albedo[3];
    int nlights;
    DevLight lights[4];
    int stream;           // 1: sample values from the caller's stream
    const float* ltab;    // triangle emitters: areas[ntri], cdf[ntri + 1], sum
};

// The caller's sample stream on the device (see pbg_sample_stream).
struct StreamArgs {
    const float* img;        // [count][2] raster position
    const float* dims;       // [count][ndims]
    const float* rng;        // the task RNG's draws after the sampler's
    int64_t count, nrng;
    int ndims;
    int64_t rng_base;        // path, bounces >= 3: this bounce's first draw
    const int32_t* hit_rank; // ... and each queue entry's rank among its hits
};

__global__ void raygen_kernel(RenderConst rc, StreamArgs sa, int64_t n, float4* __restrict__ o4,
                              float4* __restrict__ d4, int32_t* __restrict__ qidx, float* __restrict__ L,
                              float* __restrict__ beta) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    float ix, iy;
    if (rc.stream) {
        ix = sa.img[2 * s];
        iy = sa.img[2 * s + 1];
    } else {
        const int64_t pix = s / rc.spp;
        const int k = (int)(s % rc.spp);
        const int px = (int)(pix % rc.xres), py = (int)(pix / rc.xres);
        const int sx = k % rc.spp_x, sy = k / rc.spp_x;
        const float jx = rc.jitter ? rnd(rc.seed, (uint64_t)s, 0) : 0.5f;
        const float jy = rc.jitter ? rnd(rc.seed, (uint64_t)s, 1) : 0.5f;
        // (x + jx) * dx + xPos (samplers/stratified.cpp, StratifiedSample2D)
        ix = __fadd_rn(__fmul_rn(__fadd_rn((float)sx, jx), __frcp_rn((float)rc.spp_x)), (float)px);
        iy = __fadd_rn(__fmul_rn(__fadd_rn((float)sy, jy), __frcp_rn((float)rc.spp_y)), (float)py);
    }
    const V3 pc = xform_point(rc.r2c, v3(ix, iy, 0.f));
    const V3 dir = vnormalize(pc);
    const V3 o = xform_point(rc.c2w, v3(0.f, 0.f, 0.f));
    const V3 d = xform_vector(rc.c2w, dir);
    o4[s] = make_float4(o.x, o.y, o.z, 0.f);
    d4[s] = make_float4(d.x, d.y, d.z, INFINITY);
    qidx[s] = (int32_t)s;
    L[3 * s] = L[3 * s + 1] = L[3 * s + 2] = 0.f;
    beta[3 * s] = beta[3 * s + 1] = beta[3 * s + 2] = 1.f;
}

// Shading frame of pbrt's BSDF: nn, sn = Normalize(dpdu), tn = Cross(nn, sn).
struct Frame {
    V3 nn, sn, tn;
    __device__ V3 to_local(V3 v) const { return v3(vdot(v, sn), vdot(v, tn), vdot(v, nn)); }
    __device__ V3 to_world(V3 v) const {
        return v3(__fadd_rn(__fadd_rn(__fmul_rn(sn.x, v.x), __fmul_rn(tn.x, v.y)), __fmul_rn(nn.x, v.z)),
                  __fadd_rn(__fadd_rn(__fmul_rn(sn.y, v.x), __fmul_rn(tn.y, v.y)), __fmul_rn(nn.y, v.z)),
                  __fadd_rn(__fadd_rn(__fmul_rn(sn.z, v.x), __fmul_rn(tn.z, v.y)), __fmul_rn(nn.z, v.z)));
    }
};

__device__ __forceinline__ V3 tri_vertex(const float* v9, int k) { return v3(v9[3 * k], v9[3 * k + 1], v9[3 * k + 2]); }

// The scene triangle of an emitter's i-th ShapeSet shape: the ShapeSet
// constructor refines the mesh through a stack (todo.back(),
// core/light.cpp:106-118), so the mesh's triangles come out last first.
__device__ __forceinline__ int64_t shape_tri(int first, int n, int i) { return (int64_t)first + n - 1 - i; }

// Triangle::Intersect of one emitter triangle (shapes/trianglemesh.cpp:119-190):
// pbrt's exact test, and the hit's geometric normal.
__device__ bool emitter_hit(const float* v9, const float* uv6, V3 o, V3 d, float mint, float* t, V3* nn) {
    const V3 p1 = tri_vertex(v9, 0), e1 = vsub(tri_vertex(v9, 1), p1), e2 = vsub(tri_vertex(v9, 2), p1);
    float tt, b1, b2;
    if (!pbg_exact(p1.x, p1.y, p1.z, e1.x, e1.y, e1.z, e2.x, e2.y, e2.z, o.x, o.y, o.z, d.x, d.y, d.z, mint,
                   INFINITY, &tt, &b1, &b2))
        return false;
    *t = tt;
    *nn = hit_dg(v9, uv6, o, d, tt, b1, b2).nn;
    return true;
}

// DiffuseAreaLight::Sample_L over scene triangles (lights/diffuse.cpp:61-73):
// ShapeSet::Sample picks a triangle by its area CDF and a point on it
// (Triangle::Sample, UniformSampleTriangle), re-intersects the ray from p
// towards it with every triangle of the set (the last one hit gives the
// point and its normal), ShapeSet::Pdf sums each triangle's solid-angle pdf
// weighted by its area (core/light.cpp:137-165, core/shape.cpp:78-91).
__device__ void sample_emitter(const DevLight& lt, const float* ltab, const float* tri9, const float* uv6, V3 p,
                               float u0, float u1, float comp, V3* wi, V3* Li, float* pdf, V3* target) {
    const int n = lt.ntri;
    const float* areas = ltab + lt.tab;
    const float* cdf = areas + n;
    const float sum_area = cdf[n + 1];
    int k = 0;  // upper_bound: first CDF entry above comp
    while (k < n + 1 && !(cdf[k] > comp)) ++k;
    const int sn = k > 0 ? k - 1 : 0;
    const float* v = tri9 + 9 * shape_tri(lt.first, n, sn);
    const float su1 = __fsqrt_rn(u0);
    const float b1 = __fsub_rn(1.f, su1), b2 = __fmul_rn(u1, su1);
    const float b0 = __fsub_rn(__fsub_rn(1.f, b1), b2);
    const V3 p1 = tri_vertex(v, 0), p2 = tri_vertex(v, 1), p3 = tri_vertex(v, 2);
    const V3 pt = vadd(vadd(vmul(p1, b1), vmul(p2, b2)), vmul(p3, b0));
    V3 ns = vnormalize(vcross(vsub(p2, p1), vsub(p3, p1)));
    const V3 dir = vsub(pt, p);
    float thit = 1.f;
    for (int i = 0; i < n; ++i) {
        const int64_t tr = shape_tri(lt.first, n, i);
        float t;
        V3 nn;
        if (emitter_hit(tri9 + 9 * tr, uv6 ? uv6 + 6 * tr : nullptr, p, dir, 1e-3f, &t, &nn)) {
            thit = t;
            ns = nn;
        }
    }
    const V3 ps = vadd(p, vmul(dir, thit));
    *target = ps;
    *wi = vnormalize(vsub(ps, p));
    float acc = 0.f;
    for (int i = 0; i < n; ++i) {
        const int64_t tr = shape_tri(lt.first, n, i);
        float t, pi = 0.f;
        V3 nn;
        if (emitter_hit(tri9 + 9 * tr, uv6 ? uv6 + 6 * tr : nullptr, p, *wi, 1e-3f, &t, &nn)) {
            const V3 dv = vsub(p, vadd(p, vmul(*wi, t)));
            pi = __fdiv_rn(vdot(dv, dv), __fmul_rn(fabsf(vdot(nn, vneg(*wi))), areas[i]));
            if (isinf(pi)) pi = 0.f;
        }
        acc = __fadd_rn(acc, __fmul_rn(areas[i], pi));
    }
    *pdf = __fdiv_rn(acc, sum_area);
    *Li = vdot(ns, vneg(*wi)) > 0.f ? v3(lt.L[0], lt.L[1], lt.L[2]) : v3(0.f, 0.f, 0.f);
}

// Light sample (u0, u1, comp) of light lt at p: wi, radiance, pdf and the
// shadow segment (VisibilityTester::SetSegment, core/light.h:79-84).
__device__ __forceinline__ bool sample_light(const RenderConst& rc, const DevLight& lt, const float* tri9,
                                             const float* uv6, V3 p, float eps, float u1, float u2, float comp,
                                             V3* wi, V3* Li, float* pdf, float4* so, float4* sd) {
    V3 target;
    float eps2;
    if (lt.type == PBG_LIGHT_POINT) {
        target = v3(lt.pos[0], lt.pos[1], lt.pos[2]);
        *wi = vnormalize(vsub(target, p));
        *pdf = 1.f;
        const V3 dv = vsub(target, p);
        const float d2 = vdot(dv, dv);
        *Li = v3(__fdiv_rn(lt.I[0], d2), __fdiv_rn(lt.I[1], d2), __fdiv_rn(lt.I[2], d2));
        eps2 = 0.f;
    } else if (lt.type == PBG_LIGHT_MESH) {
        sample_emitter(lt, rc.ltab, tri9, uv6, p, u1, u2, comp, wi, Li, pdf, &target);
        eps2 = 1e-3f;
    } else {
        const V3 q0 = v3(lt.q0[0], lt.q0[1], lt.q0[2]);
        target = vadd(vadd(q0, vmul(v3(lt.e1[0], lt.e1[1], lt.e1[2]), u1)),
                      vmul(v3(lt.e3[0], lt.e3[1], lt.e3[2]), u2));
        const V3 dv = vsub(target, p);
        *wi = vnormalize(dv);
        const float d2 = vdot(dv, dv);
        const float cosl = -vdot(v3(lt.n[0], lt.n[1], lt.n[2]), *wi);
        if (!(cosl > 0.f) || !(d2 > 0.f)) return false;
        *pdf = __fdiv_rn(d2, __fmul_rn(cosl, lt.area));
        *Li = v3(lt.L[0], lt.L[1], lt.L[2]);
        eps2 = 1e-3f;
    }
    const float dist = vlen(vsub(p, target));
    const V3 dn = vmul(vsub(target, p), __frcp_rn(dist));
    *so = make_float4(p.x, p.y, p.z, eps);
    *sd = make_float4(dn.x, dn.y, dn.z, __fmul_rn(dist, __fsub_rn(1.f, eps2)));
    return true;
}

// Sample values of one vertex: the hash stream, or the caller's stream in
// the layout of pbg_sample_stream.
struct Draws {
    const RenderConst& rc;
    const StreamArgs& sa;
    int64_t s, j;
    int bounce;
    // light sample m of a directlighting vertex (hash: light-local index q)
    __device__ void direct_light(int m, int q, float* u0, float* u1, float* comp) const {
        if (rc.stream) {
            const float* v = sa.dims + s * sa.ndims + 6 * m;
            *u0 = v[0];
            *u1 = v[1];
            *comp = v[2];
        } else {
            *u0 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, 2 * q));
            *u1 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, 2 * q) + 1);
            *comp = rnd(rc.seed, (uint64_t)s, dim_extra(bounce, m));
        }
    }
    // the path integrator's light choice and light sample at this bounce
    __device__ void path_light(float* lnum, float* u0, float* u1, float* comp) const {
        if (!rc.stream) {
            *lnum = rnd(rc.seed, (uint64_t)s, dim_extra(bounce, 15));
            *u0 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, 0));
            *u1 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, 1));
            *comp = rnd(rc.seed, (uint64_t)s, dim_extra(bounce, 0));
        } else if (bounce < 3) {
            const float* v = sa.dims + s * sa.ndims + 10 * bounce;
            *lnum = v[0];
            *u0 = v[1];
            *u1 = v[2];
            *comp = v[3];
        } else {
            const float* v = sa.rng + sa.rng_base + 7 * s;
            *lnum = v[0];
            *u0 = v[1];
            *u1 = v[2];
            *comp = v[3];
        }
    }
    // the path's BSDF sample (uDir) and Russian roulette value
    __device__ void path_bsdf(float* u0, float* u1) const {
        if (!rc.stream) {
            *u0 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, kDimBsdf));
            *u1 = rnd(rc.seed, (uint64_t)s, dim_of(bounce, kDimBsdf + 1));
        } else if (bounce < 3) {
            const float* v = sa.dims + s * sa.ndims + 10 * bounce;
            *u0 = v[7];
            *u1 = v[8];
        } else {
            const float* v = sa.rng + sa.rng_base + 7 * sa.count + (int64_t)sa.hit_rank[j] * (bounce > 3 ? 4 : 3);
            *u0 = v[0];
            *u1 = v[1];
        }
    }
    __device__ float path_rr() const {
        if (!rc.stream) return rnd(rc.seed, (uint64_t)s, dim_of(bounce, kDimRR));
        return sa.rng[sa.rng_base + 7 * sa.count + (int64_t)sa.hit_rank[j] * 4 + 3];
    }
};

// Where a bounce's rays come from and go: the queue being shaded (its length
// read on the device where the host does not know it) and the queues that its
// shadow and bounce rays are appended to.
struct ShadeIO {
    int64_t nq;
    const uint32_t* nq_dev;  // NULL: nq entries
    const int32_t* qidx;
    const float4 *qo, *qd;
    const int32_t* prim;
    const float *th, *b1, *b2;
    float4 *so, *sd;         // shadow rays (stream renders: by slot)
    int32_t* spos;           // each slot's place among them, -1: none
    uint32_t* nshadow;
    int32_t* nidx;           // the next bounce's queue (stream renders: rays by entry, no nidx)
    float4 *no, *nd;
    uint32_t* nnext;
    uint8_t *sflag, *nflag;  // stream renders: which slots and entries hold a ray
    float* scontrib;
    float* emit;             // camera hits on emitting triangles (NULL: none at this bounce)
};

__device__ __forceinline__ int64_t queue_length(int64_t n, const uint32_t* dev) { return dev ? (int64_t)*dev : n; }

// The block's items get consecutive places in a queue, in thread order, behind
// one atomic.  Every thread of the block calls it.
constexpr int kShadeThreads = 128;
__device__ __forceinline__ uint32_t block_place(uint32_t in_warp, uint32_t warp_total, uint32_t* count) {
    __shared__ uint32_t wcount[kShadeThreads / 32], base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) wcount[warp] = warp_total;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kShadeThreads / 32; ++w) {
        before += w < warp ? wcount[w] : 0u;
        total += wcount[w];
    }
    if (threadIdx.x == 0 && total) base = atomicAdd(count, total);
    __syncthreads();
    return base + before + in_warp;
}
__device__ __forceinline__ uint32_t block_append(bool has, uint32_t* count) {
    const unsigned b = __ballot_sync(0xffffffffu, has);
    return block_place(__popc(b & ((1u << (threadIdx.x & 31)) - 1u)), __popc(b), count);
}
// The same for a number of items per thread, kept together.
__device__ __forceinline__ uint32_t block_append_n(uint32_t n, uint32_t* count) {
    uint32_t incl = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, off);
        if ((threadIdx.x & 31) >= off) incl += x;
    }
    return block_place(incl - n, __shfl_sync(0xffffffffu, incl, 31), count);
}

// A shaded hit.
struct Vertex {
    V3 p, ng, wo, wol, fR, bt;
    Frame fr;
    float won, eps;
};

// The direct lighting of one light sample at v: the shadow ray and what it
// carries if unoccluded; false when it carries nothing.
__device__ __forceinline__ bool light_ray(const RenderConst& rc, const DevLight& lt, const float* tri9, const float* uv6,
                                          const Vertex& v, float u1, float u2, float comp, float4* o_, float4* d_, V3* out) {
    V3 wi, Li;
    float pdf;
    if (!sample_light(rc, lt, tri9, uv6, v.p, v.eps, u1, u2, comp, &wi, &Li, &pdf, o_, d_)) return false;
    if (!(pdf > 0.f) || (Li.x == 0.f && Li.y == 0.f && Li.z == 0.f)) return false;
    const bool refl = __fmul_rn(vdot(wi, v.ng), v.won) > 0.f;
    if (!refl) return false;  // f = 0: Lambertian reflects only
    const bool all = rc.integrator == PBG_INTEGRATOR_DIRECT;
    const float absdot = fabsf(vdot(wi, v.fr.nn));
    const V3 fL = v3(__fmul_rn(v.fR.x, Li.x), __fmul_rn(v.fR.y, Li.y), __fmul_rn(v.fR.z, Li.z));
    V3 c;
    if (lt.type == PBG_LIGHT_POINT) {
        if (all) {  // f * Li * AbsDot / lightPdf
            c = v3(__fdiv_rn(__fmul_rn(fL.x, absdot), pdf), __fdiv_rn(__fmul_rn(fL.y, absdot), pdf),
                   __fdiv_rn(__fmul_rn(fL.z, absdot), pdf));
        } else {    // f * Li * (AbsDot / lightPdf)
            const float w = __fdiv_rn(absdot, pdf);
            c = v3(__fmul_rn(fL.x, w), __fmul_rn(fL.y, w), __fmul_rn(fL.z, w));
        }
    } else {
        const V3 wil = v.fr.to_local(wi);
        const bool same = __fmul_rn(v.wol.z, wil.z) > 0.f;
        const float bpdf = same ? __fmul_rn(fabsf(wil.z), kInvPi) : 0.f;
        // PowerHeuristic(1, pdf, 1, bpdf)
        const float f2 = __fmul_rn(pdf, pdf), g2 = __fmul_rn(bpdf, bpdf);
        const float weight = __fdiv_rn(f2, __fadd_rn(f2, g2));
        if (all) {  // f * Li * AbsDot * weight / lightPdf
            c = v3(__fdiv_rn(__fmul_rn(__fmul_rn(fL.x, absdot), weight), pdf),
                   __fdiv_rn(__fmul_rn(__fmul_rn(fL.y, absdot), weight), pdf),
                   __fdiv_rn(__fmul_rn(__fmul_rn(fL.z, absdot), weight), pdf));
        } else {    // f * Li * (AbsDot * weight / lightPdf)
            const float w = __fdiv_rn(__fmul_rn(absdot, weight), pdf);
            c = v3(__fmul_rn(fL.x, w), __fmul_rn(fL.y, w), __fmul_rn(fL.z, w));
        }
    }
    if (!all) {  // Ld *= nLights, then L += pathThroughput * Ld
        const float fl = (float)rc.nlights;
        c = v3(__fmul_rn(c.x, fl), __fmul_rn(c.y, fl), __fmul_rn(c.z, fl));
        c = v3(__fmul_rn(v.bt.x, c.x), __fmul_rn(v.bt.y, c.y), __fmul_rn(v.bt.z, c.z));
    }
    *out = c;
    return true;
}

// BSDF sample for the next vertex (Lambertian::Sample_f, cosine-weighted
// through ConcentricSampleDisk, core/montecarlo.cpp): the direction and the
// new throughput; false when the path ends here.
__device__ __forceinline__ bool bounce_dir(const RenderConst& rc, const Draws& dr, int bounce, const Vertex& v, int* rstat,
                                           V3* wi_out, V3* nb_out) {
    float u1, u2;
    dr.path_bsdf(&u1, &u2);
    float sx = __fsub_rn(__fmul_rn(2.f, u1), 1.f), sy = __fsub_rn(__fmul_rn(2.f, u2), 1.f);
    float dx = 0.f, dy = 0.f;
    if (!(sx == 0.f && sy == 0.f)) {
        float r, theta;
        if (sx >= -sy) {
            if (sx > sy) {
                r = sx;
                theta = sy > 0.f ? __fdiv_rn(sy, r) : __fadd_rn(8.f, __fdiv_rn(sy, r));
            } else {
                r = sy;
                theta = __fsub_rn(2.f, __fdiv_rn(sx, r));
            }
        } else {
            if (sx <= sy) {
                r = -sx;
                theta = __fsub_rn(4.f, __fdiv_rn(sy, r));
            } else {
                r = -sy;
                theta = __fadd_rn(6.f, __fdiv_rn(sx, r));
            }
        }
        float st, ct;
        if (rc.stream) {
            // theta *= M_PI / 4.f is a double product rounded to float; the
            // reference's cosf/sinf come from the host's libm, here the
            // correctly rounded value (one double evaluation, rounded once)
            theta = __double2float_rn(__dmul_rn((double)theta, 0.78539816339744830962));
            double ds, dc;
            sincos((double)theta, &ds, &dc);
            st = __double2float_rn(ds);
            ct = __double2float_rn(dc);
        } else {
            theta = __fmul_rn(theta, 0.785398163397448309616f);
            own_sincos(theta, &st, &ct);
        }
        dx = __fmul_rn(r, ct);
        dy = __fmul_rn(r, st);
    }
    V3 wil = v3(dx, dy, __fsqrt_rn(fmaxf(0.f, __fsub_rn(__fsub_rn(1.f, __fmul_rn(dx, dx)), __fmul_rn(dy, dy)))));
    if (v.wol.z < 0.f) wil.z = -wil.z;
    const bool same = __fmul_rn(v.wol.z, wil.z) > 0.f;
    const float pdf = same ? __fmul_rn(fabsf(wil.z), kInvPi) : 0.f;
    const V3 wi = v.fr.to_world(wil);
    const bool refl = __fmul_rn(vdot(wi, v.ng), v.won) > 0.f;
    if (!refl || !(pdf > 0.f)) {
        // the reference keeps such a ray alive with its old direction
        // (integrators/path.cpp:112-113); a stream render stops matching it
        if (rc.stream) atomicAdd(&rstat[0], 1);
        return false;
    }
    const float absdot = fabsf(vdot(wi, v.fr.nn));
    // pathThroughput *= f * AbsDot(wi, n) / pdf
    V3 nb = v3(__fmul_rn(v.bt.x, __fdiv_rn(__fmul_rn(v.fR.x, absdot), pdf)),
               __fmul_rn(v.bt.y, __fdiv_rn(__fmul_rn(v.fR.y, absdot), pdf)),
               __fmul_rn(v.bt.z, __fdiv_rn(__fmul_rn(v.fR.z, absdot), pdf)));
    if (bounce > 3) {  // Russian roulette (integrators/path.cpp:117-124)
        const float y = __fadd_rn(__fadd_rn(__fmul_rn(0.212671f, nb.x), __fmul_rn(0.715160f, nb.y)),
                                  __fmul_rn(0.072169f, nb.z));
        const float cont = fminf(0.5f, y);
        if (dr.path_rr() > cont) return false;
        nb = v3(__fdiv_rn(nb.x, cont), __fdiv_rn(nb.y, cont), __fdiv_rn(nb.z, cont));
    }
    if (bounce == rc.max_depth) return false;
    *wi_out = wi;
    *nb_out = nb;
    return true;
}

// One queue entry: shade the hit, append its shadow rays and its bounce ray,
// note its emission (camera hits on emitting triangles).  A gather-bound
// kernel: 6 CTAs per SM measured best of 4, 5, 6 and 8 on the path frame
// (20.37 / 20.12 / 20.02 / 20.25 ms).  Appending here replaced slot arrays,
// two counting passes, six scan kernels, two compaction passes and two host
// reads per bounce: 211 x 157 path preview 1,191 -> 650 us, 1024 x 1024 x 8
// path frame 20.7 -> 20.0 ms.  directlighting keeps a hit's shadow rays
// together, four at a time through shared memory: slot by slot they lie 32
// pixels apart in a warp and the walk of a four-sample still takes 60 us more.
constexpr int kShadeMinBlocks = 6;
constexpr int kShadeChunk = 4;
template <bool STREAM, bool DIRECT>
__global__ void __launch_bounds__(kShadeThreads, kShadeMinBlocks)
    shade_kernel(RenderConst rc, StreamArgs sa, int bounce, ShadeIO io, const float* __restrict__ tri9,
                 const float* __restrict__ uv6, float* __restrict__ beta, int kslots, int* __restrict__ rstat) {
    const int64_t nq = queue_length(io.nq, io.nq_dev);
    // whole blocks: every thread takes part in each append
    for (int64_t j0 = (int64_t)blockIdx.x * kShadeThreads; j0 < nq; j0 += (int64_t)gridDim.x * kShadeThreads) {
        const int64_t j = j0 + threadIdx.x;
        const bool in = j < nq;
        const int32_t pr = in ? io.prim[j] : -1;
        const bool hit = pr >= 0;  // a miss: no environment light
        const int64_t s = hit ? io.qidx[j] : 0;
        const Draws dr{rc, sa, s, j, bounce};
        Vertex v{};
        V3 emit = v3(0.f, 0.f, 0.f);
        if (hit) {
            const float4 o4 = io.qo[j], d4 = io.qd[j];
            const V3 ro = v3(o4.x, o4.y, o4.z), rdir = v3(d4.x, d4.y, d4.z);
            const float t = io.th[j];
            const HitDG g = hit_dg(tri9 + 9 * (int64_t)pr, uv6 ? uv6 + 6 * (int64_t)pr : nullptr, ro, rdir, t,
                                   io.b1[j], io.b2[j]);
            v.p = g.p;
            v.eps = __fmul_rn(1e-3f, t);  // rayEpsilon (shapes/trianglemesh.cpp:190)
            v.fr.nn = g.nn;
            v.fr.sn = vnormalize(g.dpdu);
            v.fr.tn = vcross(v.fr.nn, v.fr.sn);
            v.ng = g.nn;
            v.wo = vneg(rdir);
            // Intersection::Le at camera hits (DiffuseAreaLight::L, lights/diffuse.h:43-45)
            if (io.emit) {
                for (int l = 0; l < rc.nlights; ++l) {
                    const DevLight& lt = rc.lights[l];
                    if (lt.type == PBG_LIGHT_MESH && pr >= lt.first && pr < lt.first + lt.ntri && vdot(g.nn, v.wo) > 0.f)
                        emit = v3(lt.L[0], lt.L[1], lt.L[2]);
                }
            }
            v.fR = v3(__fmul_rn(rc.albedo[0], kInvPi), __fmul_rn(rc.albedo[1], kInvPi), __fmul_rn(rc.albedo[2], kInvPi));
            v.bt = v3(beta[3 * s], beta[3 * s + 1], beta[3 * s + 2]);
            v.won = vdot(v.wo, v.ng);
            v.wol = v.fr.to_local(v.wo);
        }
        if (io.emit && in) {
            io.emit[3 * j] = emit.x;
            io.emit[3 * j + 1] = emit.y;
            io.emit[3 * j + 2] = emit.z;
        }

        // Direct lighting: every light and sample (directlighting) or one
        // light sample (path).
        auto put_contrib = [&](int slot, const V3& c) {
            float* w = io.scontrib + 3 * (j * kslots + slot);
            w[0] = c.x;
            w[1] = c.y;
            w[2] = c.z;
        };
        auto put_shadow = [&](int slot, bool has, int64_t at, const float4& o_, const float4& d_) {
            const int64_t si = j * kslots + slot;
            if (STREAM) {
                if (in) io.sflag[si] = has ? 1 : 0;
                at = si;
            } else if (in) {
                io.spos[si] = has ? (int32_t)at : -1;
            }
            if (!has) return;
            io.so[at] = o_;
            io.sd[at] = d_;
        };
        float4 o_ = make_float4(0.f, 0.f, 0.f, 0.f), d_ = o_;
        V3 c = v3(0.f, 0.f, 0.f);
        int slot = 0;
        if (DIRECT && rc.nlights > 0) {
            __shared__ float4 ray_of[STREAM || !DIRECT ? 1 : 2 * kShadeChunk * kShadeThreads];
            uint32_t held = 0;  // this chunk's slots that have a ray
            int first = 0;      // its first slot
            auto flush = [&]() {  // a chunk's rays to the queue, thread by thread
                uint32_t at = block_append_n(__popc(held), io.nshadow);
                for (int k = 0; first < slot; ++first, ++k) {
                    const bool has = (held >> k & 1u) != 0;
                    const int e = k * kShadeThreads + threadIdx.x;
                    if (has) {
                        o_ = ray_of[2 * e];
                        d_ = ray_of[2 * e + 1];
                    }
                    put_shadow(first, has, at, o_, d_);
                    at += has ? 1u : 0u;
                }
                held = 0;
            };
            for (int l = 0; l < rc.nlights; ++l) {
                const DevLight& lt = rc.lights[l];
                const int ns = lt.type == PBG_LIGHT_POINT ? 1 : max(lt.nsamples, 1);
                for (int q = 0; q < ns && slot < kslots; ++q) {
                    bool has = false;
                    if (hit) {
                        float u1, u2, comp;
                        dr.direct_light(slot, q, &u1, &u2, &comp);
                        has = light_ray(rc, lt, tri9, uv6, v, u1, u2, comp, &o_, &d_, &c);
                    }
                    if (has) put_contrib(slot, c);
                    if (STREAM) {
                        put_shadow(slot++, has, 0, o_, d_);
                        continue;
                    }
                    if (has) {
                        const int e = (slot - first) * kShadeThreads + threadIdx.x;
                        ray_of[2 * e] = o_;
                        ray_of[2 * e + 1] = d_;
                        held |= 1u << (slot - first);
                    }
                    ++slot;
                    if (slot - first == kShadeChunk) flush();
                }
            }
            if (!STREAM && first < slot) flush();
        } else if (!DIRECT && rc.nlights > 0) {
            bool has = false;
            if (hit) {
                // UniformSampleOneLight: lightNum = min(Floor2Int(u * nLights), nLights - 1)
                float lnum, u1, u2, comp;
                dr.path_light(&lnum, &u1, &u2, &comp);
                const int l = min((int)floorf(__fmul_rn(lnum, (float)rc.nlights)), rc.nlights - 1);
                has = light_ray(rc, rc.lights[l], tri9, uv6, v, u1, u2, comp, &o_, &d_, &c);
            }
            if (has) put_contrib(0, c);
            put_shadow(0, has, STREAM ? 0 : (int64_t)block_append(has, io.nshadow), o_, d_);
            slot = 1;
        }
        for (; slot < kslots; ++slot) put_shadow(slot, false, 0, o_, d_);  // no lights
        if (DIRECT) continue;

        V3 wi = v3(0.f, 0.f, 0.f), nb = wi;
        const bool go = hit && bounce_dir(rc, dr, bounce, v, rstat, &wi, &nb);
        int64_t at = j;
        if (STREAM) {
            if (in) io.nflag[j] = go ? 1 : 0;
        } else {
            at = (int64_t)block_append(go, io.nnext);
        }
        if (go) {
            beta[3 * s] = nb.x;
            beta[3 * s + 1] = nb.y;
            beta[3 * s + 2] = nb.z;
            if (!STREAM) io.nidx[at] = (int32_t)s;
            io.no[at] = make_float4(v.p.x, v.p.y, v.p.z, v.eps);
            io.nd[at] = make_float4(wi.x, wi.y, wi.z, INFINITY);
        }
    }
}

// Triangle-emitter tables: Triangle::Area (shapes/trianglemesh.cpp:276-282)
// in ShapeSet order, the total area and the Distribution1D CDF
// (core/montecarlo.h:48-70), in pbrt's float arithmetic.  One thread.
__global__ void emitter_setup_kernel(const float* __restrict__ tri9, int first, int n, float* __restrict__ tab) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    float sum = 0.f;
    for (int i = 0; i < n; ++i) {
        const float* v = tri9 + 9 * shape_tri(first, n, i);
        const V3 p1 = tri_vertex(v, 0);
        const V3 c = vcross(vsub(tri_vertex(v, 1), p1), vsub(tri_vertex(v, 2), p1));
        const float a = __fmul_rn(0.5f, vlen(c));
        tab[i] = a;
        sum = __fadd_rn(sum, a);
    }
    float* cdf = tab + n;
    cdf[0] = 0.f;
    for (int i = 1; i <= n; ++i) cdf[i] = __fadd_rn(cdf[i - 1], __fdiv_rn(tab[i - 1], (float)n));
    const float integral = cdf[n];
    for (int i = 1; i <= n; ++i)
        cdf[i] = integral == 0.f ? __fdiv_rn((float)i, (float)n) : __fdiv_rn(cdf[i], integral);
    cdf[n + 1] = sum;
}

// Order-preserving compaction, phase 1: per-block count of set flags.
__global__ void flag_count_kernel(const uint8_t* __restrict__ flag, int64_t n, uint32_t* __restrict__ counts) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int c = __syncthreads_count(i < n && flag[i] != 0);
    if (threadIdx.x == 0) counts[blockIdx.x] = (uint32_t)c;
}

// Phase 2 (after a scan of the block counts): rank inside the block from
// warp ballots, then gather.  pos[i] receives the dense index or -1.
template <typename Fn>
__device__ __forceinline__ void compact_rank(const uint8_t* flag, int64_t n, const uint32_t* offs,
                                             int32_t* pos, Fn&& emit) {
    __shared__ uint32_t warp_base[32];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool f = i < n && flag[i] != 0;
    const unsigned b = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) warp_base[warp] = __popc(b);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            const uint32_t c = warp_base[w];
            warp_base[w] = run;
            run += c;
        }
    }
    __syncthreads();
    if (i >= n) return;
    if (!f) {
        if (pos) pos[i] = -1;
        return;
    }
    const uint32_t dst = offs[blockIdx.x] + warp_base[warp] + __popc(b & ((1u << lane) - 1u));
    if (pos) pos[i] = (int32_t)dst;
    emit(i, dst);
}

__global__ void compact_shadow_kernel(const uint8_t* __restrict__ flag, int64_t n,
                                      const uint32_t* __restrict__ offs, const float4* __restrict__ so,
                                      const float4* __restrict__ sd, float4* __restrict__ qo,
                                      float4* __restrict__ qd, int32_t* __restrict__ pos) {
    compact_rank(flag, n, offs, pos, [&](int64_t i, uint32_t dst) {
        qo[dst] = so[i];
        qd[dst] = sd[i];
    });
}

__global__ void compact_bounce_kernel(const uint8_t* __restrict__ flag, int64_t n,
                                      const uint32_t* __restrict__ offs, const int32_t* __restrict__ qidx,
                                      const float4* __restrict__ no, const float4* __restrict__ nd_,
                                      int32_t* __restrict__ qidx_out, float4* __restrict__ qo,
                                      float4* __restrict__ qd) {
    compact_rank(flag, n, offs, nullptr, [&](int64_t i, uint32_t dst) {
        qidx_out[dst] = qidx[i];
        qo[dst] = no[i];
        qd[dst] = nd_[i];
    });
}

// Stream renders, path bounces >= 3: each queue entry's rank among the
// entries that hit (the order in which the reference's BSDF loop draws).
__global__ void hit_flag_kernel(const int32_t* __restrict__ prim, int64_t n, uint8_t* __restrict__ flag) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flag[i] = prim[i] >= 0 ? 1 : 0;
}

__global__ void hit_rank_kernel(const uint8_t* __restrict__ flag, int64_t n, const uint32_t* __restrict__ offs,
                                int32_t* __restrict__ rank) {
    compact_rank(flag, n, offs, rank, [](int64_t, uint32_t) {});
}

// Unoccluded shadow contributions and emission (emit NULL: zero), added per
// entry in slot order.  directlighting: Ld = the sum over every light and sample
// (UniformSampleAllLights' batch form, core/integrator.cpp:73-122, does not
// divide by the sample count), L += Ld, then L += Le
// (integrators/directlighting.cpp:112-133); path: L += Le at the camera
// vertex, then the single slot, which already carries beta * nLights * Ld.
__global__ void resolve_kernel(RenderConst rc, int64_t n, const uint32_t* __restrict__ n_dev, int kslots,
                               const int32_t* __restrict__ qidx, const int32_t* __restrict__ spos,
                               const uint8_t* __restrict__ occ, const float* __restrict__ scontrib,
                               const float* __restrict__ emit, float* __restrict__ L) {
    const int64_t nq = queue_length(n, n_dev);
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nq; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = qidx[j];
        V3 e = v3(0.f, 0.f, 0.f), a = e;
        if (emit) e = v3(emit[3 * j], emit[3 * j + 1], emit[3 * j + 2]);
        V3 l = v3(L[3 * s], L[3 * s + 1], L[3 * s + 2]);
        const bool direct = rc.integrator == PBG_INTEGRATOR_DIRECT;
        if (!direct) a = vadd(l, e);
        for (int k = 0; k < kslots; ++k) {
            const int64_t si = j * kslots + k;
            const int32_t at = spos[si];
            if (at < 0 || occ[at]) continue;
            a = vadd(a, v3(scontrib[3 * si], scontrib[3 * si + 1], scontrib[3 * si + 2]));
        }
        l = direct ? vadd(vadd(l, a), e) : a;
        L[3 * s] = l.x;
        L[3 * s + 1] = l.y;
        L[3 * s + 2] = l.z;
    }
}

// ImageFilm: RGB -> XYZ per sample, summed in sample order, back to RGB,
// divided by the weight sum, clamped at zero (film/image.cpp).  A sample
// whose radiance breadthFirst::Li rejects (NaN, luminance below -1e-5 or
// infinite, renderers/breadth-first.cpp:196-213) adds black.  Samples of
// pixel p: [off[p], off[p + 1]) of idx when a list is given (stream
// renders), else the spp consecutive samples p * spp ...
__device__ __forceinline__ void film_add(const float* L, int64_t s, float* X, float* Y, float* Z, float* w) {
    float r = L[3 * s], g = L[3 * s + 1], b = L[3 * s + 2];
    const float lum = __fadd_rn(__fadd_rn(__fmul_rn(0.212671f, r), __fmul_rn(0.715160f, g)), __fmul_rn(0.072169f, b));
    if (isnan(r) || isnan(g) || isnan(b) || lum < -1e-5f || isinf(lum)) r = g = b = 0.f;
    const float x = __fadd_rn(__fadd_rn(__fmul_rn(0.412453f, r), __fmul_rn(0.357580f, g)), __fmul_rn(0.180423f, b));
    const float y = __fadd_rn(__fadd_rn(__fmul_rn(0.212671f, r), __fmul_rn(0.715160f, g)), __fmul_rn(0.072169f, b));
    const float z = __fadd_rn(__fadd_rn(__fmul_rn(0.019334f, r), __fmul_rn(0.119193f, g)), __fmul_rn(0.950227f, b));
    *X = __fadd_rn(*X, x);
    *Y = __fadd_rn(*Y, y);
    *Z = __fadd_rn(*Z, z);
    *w = __fadd_rn(*w, 1.f);
}

__global__ void film_kernel(int64_t npix, int spp, const int32_t* __restrict__ off, const int32_t* __restrict__ idx,
                            const float* __restrict__ L, float* __restrict__ rgb) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float X = 0.f, Y = 0.f, Z = 0.f, w = 0.f;
    if (off) {
        for (int32_t k = off[p]; k < off[p + 1]; ++k) film_add(L, idx[k], &X, &Y, &Z, &w);
    } else {
        for (int k = 0; k < spp; ++k) film_add(L, p * spp + k, &X, &Y, &Z, &w);
    }
    float R = __fsub_rn(__fsub_rn(__fmul_rn(3.240479f, X), __fmul_rn(1.537150f, Y)), __fmul_rn(0.498535f, Z));
    float G = __fadd_rn(__fadd_rn(__fmul_rn(-0.969256f, X), __fmul_rn(1.875991f, Y)), __fmul_rn(0.041556f, Z));
    float B = __fadd_rn(__fsub_rn(__fmul_rn(0.055648f, X), __fmul_rn(0.204043f, Y)), __fmul_rn(1.057311f, Z));
    if (w != 0.f) {
        const float inv = __frcp_rn(w);
        R = fmaxf(0.f, __fmul_rn(R, inv));
        G = fmaxf(0.f, __fmul_rn(G, inv));
        B = fmaxf(0.f, __fmul_rn(B, inv));
    }
    rgb[3 * p] = R;
    rgb[3 * p + 1] = G;
    rgb[3 * p + 2] = B;
}

// ------------------------------------------------------------------ host

int scan_counts(pbg_scene* s, uint32_t* a, int64_t m, cudaStream_t st);

// One bounce's shadow queue: its rays, their occlusion, each slot's place and
// contribution, the bounce's emission.  Path frames on ray-bvh and naive
// scenes keep two, so that a bounce's shadow traversal and resolve run on a
// second stream beside the next bounce's nearest-hit traversal.  so / sd /
// sflag: stream renders' slots before their ordered compaction.
struct ShadowSet {
    DeviceBuffer so, sd, scontrib, sflag, spos, sqo, sqd, occ, emit;
    void release_all() {
        DeviceBuffer* all[] = {&so, &sd, &scontrib, &sflag, &spos, &sqo, &sqd, &occ, &emit};
        for (DeviceBuffer* b : all) release(*b);
    }
};

// A bounce's queue lengths and walk counters on the device, zeroed together
// for kCountedBounces bounces at a time.
struct BounceCount {
    uint32_t nshadow, nnext;
    unsigned long long next_near, next_any, pad;
};
static_assert(sizeof(BounceCount) == 32, "two words, two counters");
constexpr int kCountedBounces = 8;

struct RenderBuffers {
    DeviceBuffer o4, d4, qidx[3], L, beta, prim, t, b1, b2, no, nd, nflag, o42, d42, counts, rgb, rstat,
        ltab, simg, sdims, srng, hflag, hrank, foff, fidx, bcount;
    ShadowSet sh[2];
    cudaStream_t side = nullptr;           // the shadow stream of overlapped frames
    cudaEvent_t ready[2] = {}, resolved[2] = {}, span[2] = {};
    struct HostWords {                     // pinned: what the host reads of a frame
        BounceCount count[kCountedBounces];
        int rstat[4], status[4];
    }* words = nullptr;
    ~RenderBuffers() {
        DeviceBuffer* all[] = {&o4,   &d4,    &qidx[0], &qidx[1], &qidx[2], &L,    &beta, &prim,  &t,
                               &b1,   &b2,    &no,      &nd,      &nflag,   &o42,  &d42,  &counts, &rgb,
                               &rstat, &ltab, &simg,    &sdims,   &srng,    &hflag, &hrank, &foff, &fidx,
                               &bcount};
        for (DeviceBuffer* b : all) release(*b);
        for (ShadowSet& x : sh) x.release_all();
        for (int k = 0; k < 2; ++k) {
            if (ready[k]) cudaEventDestroy(ready[k]);
            if (resolved[k]) cudaEventDestroy(resolved[k]);
            if (span[k]) cudaEventDestroy(span[k]);
        }
        if (side) cudaStreamDestroy(side);
        if (words) cudaFreeHost(words);
    }
};

void render_free(pbg_scene* s) {
    delete s->render_bufs;
    s->render_bufs = nullptr;
}

static int compact_count(pbg_scene* s, const uint8_t* flag, int64_t n, uint32_t* counts, int64_t* total,
                         cudaStream_t st) {
    const int64_t blocks = (n + 255) / 256;
    flag_count_kernel<<<(unsigned)blocks, 256, 0, st>>>(flag, n, counts);
    PBG_CUDA(cudaGetLastError());
    uint32_t last_count = 0;
    PBG_CUDA(cudaMemcpyAsync(&last_count, counts + blocks - 1, 4, cudaMemcpyDeviceToHost, st));
    int rc = scan_counts(s, counts, blocks, st);
    if (rc) return rc;
    uint32_t last_off = 0;
    PBG_CUDA(cudaMemcpyAsync(&last_off, counts + blocks - 1, 4, cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaStreamSynchronize(st));
    *total = (int64_t)last_off + last_count;
    s->counters.kernel_launches += 1;
    return PBG_OK;
}

// The pixels a sample at (x, y) adds to: ImageFilm::AddSample's footprint of
// the box filter of radius 0.5 (film/image.cpp), clipped to the image.
static void film_footprint(float x, float y, int xres, int yres, int* x0, int* x1, int* y0, int* y1) {
    const float dx = x - 0.5f, dy = y - 0.5f;
    *x0 = std::max((int)std::ceil(dx - 0.5f), 0);
    *x1 = std::min((int)std::floor(dx + 0.5f), xres - 1);
    *y0 = std::max((int)std::ceil(dy - 0.5f), 0);
    *y1 = std::min((int)std::floor(dy + 0.5f), yres - 1);
}

int render(pbg_scene* s, const pbg_camera* cam, const pbg_light* lights, int32_t nlights,
           const pbg_render_params* prm, const pbg_sample_stream* stream, float* rgb_host,
           pbg_render_stats* stats) {
    if (!cam || !prm || nlights < 0 || nlights > 4 || (nlights > 0 && !lights) || !rgb_host ||
        cam->xres <= 0 || cam->yres <= 0 || prm->spp_x <= 0 || prm->spp_y <= 0 ||
        (prm->integrator != PBG_INTEGRATOR_DIRECT && prm->integrator != PBG_INTEGRATOR_PATH)) {
        set_last_error("pbg_render: bad arguments");
        return PBG_ERR_INVALID_ARGUMENT;
    }
    RenderConst rc{};
    memcpy(rc.r2c, cam->raster_to_camera, sizeof(rc.r2c));
    memcpy(rc.c2w, cam->camera_to_world, sizeof(rc.c2w));
    rc.xres = cam->xres;
    rc.yres = cam->yres;
    rc.spp_x = prm->spp_x;
    rc.spp_y = prm->spp_y;
    rc.spp = prm->spp_x * prm->spp_y;
    rc.jitter = prm->jitter;
    rc.max_depth = prm->max_depth > 0 ? prm->max_depth : 5;
    rc.integrator = prm->integrator;
    rc.seed = prm->seed;
    rc.stream = stream != nullptr;
    for (int k = 0; k < 3; ++k) rc.albedo[k] = prm->albedo[k];
    rc.nlights = nlights;
    int kslots = 0, ltab_floats = 0;
    for (int l = 0; l < nlights; ++l) {
        const pbg_light& in = lights[l];
        DevLight& d = rc.lights[l];
        d.type = in.type;
        d.nsamples = in.nsamples > 0 ? in.nsamples : 1;
        for (int k = 0; k < 3; ++k) {
            d.pos[k] = in.pos[k];
            d.I[k] = in.intensity[k];
            d.q0[k] = in.quad[k];
            d.e1[k] = in.quad[3 + k] - in.quad[k];
            d.e3[k] = in.quad[9 + k] - in.quad[k];
            d.L[k] = in.radiance[k];
        }
        if (in.type == PBG_LIGHT_MESH) {
            if (in.ntri <= 0 || in.ntri > 64 || in.first_tri < 0 || (int64_t)in.first_tri + in.ntri > s->ntri) {
                set_last_error("pbg_render: a triangle emitter needs 1..64 triangles of the scene");
                return PBG_ERR_INVALID_ARGUMENT;
            }
            d.first = in.first_tri;
            d.ntri = in.ntri;
            d.tab = ltab_floats;
            ltab_floats += 2 * in.ntri + 2;
        } else if (in.type != PBG_LIGHT_POINT && in.type != PBG_LIGHT_QUAD) {
            set_last_error("pbg_render: unknown light type");
            return PBG_ERR_INVALID_ARGUMENT;
        }
        const double cx = (double)d.e1[1] * d.e3[2] - (double)d.e1[2] * d.e3[1];
        const double cy = (double)d.e1[2] * d.e3[0] - (double)d.e1[0] * d.e3[2];
        const double cz = (double)d.e1[0] * d.e3[1] - (double)d.e1[1] * d.e3[0];
        const double len = std::sqrt(cx * cx + cy * cy + cz * cz);
        d.area = (float)len;
        d.n[0] = len > 0 ? (float)(cx / len) : 0.f;
        d.n[1] = len > 0 ? (float)(cy / len) : 0.f;
        d.n[2] = len > 0 ? (float)(cz / len) : 0.f;
        if (prm->integrator == PBG_INTEGRATOR_DIRECT)
            kslots += d.type == PBG_LIGHT_POINT ? 1 : d.nsamples;
        else if (l == 0)
            kslots = 1;
    }
    if (kslots == 0) kslots = 1;
    const int64_t npix = (int64_t)cam->xres * cam->yres;
    const int64_t n = stream ? stream->count : npix * rc.spp;
    if (n <= 0 || n > (int64_t)INT32_MAX / std::max(kslots, 1)) {
        set_last_error("pbg_render: image too large for one batch, or an empty sample stream");
        return PBG_ERR_INVALID_ARGUMENT;
    }
    if (stream) {
        const int need = prm->integrator == PBG_INTEGRATOR_PATH ? 30 : 6 * kslots;
        if (!stream->image_xy || !stream->dims || stream->ndims < need || stream->nrng < 0 ||
            (stream->nrng > 0 && !stream->rng)) {
            set_last_error("pbg_render_stream: the stream needs image positions, the sample values of its layout "
                           "(30 per sample for path, 6 per light sample for directlighting) and its RNG draws");
            return PBG_ERR_INVALID_ARGUMENT;
        }
    }
    cudaStream_t st = s->stream;
    if (!s->render_bufs) s->render_bufs = new RenderBuffers();
    RenderBuffers& B = *s->render_bufs;  // grown on demand, kept for the next frame
    int r;
    const size_t nk = (size_t)n * kslots;
    bool emitters = false;
    for (int l = 0; l < nlights; ++l) emitters = emitters || rc.lights[l].type == PBG_LIGHT_MESH;
    // Overlapped bounces (path frames on ray-bvh and naive scenes): each
    // bounce's shadow traversal and resolve go to a second stream, beside
    // the next bounce's nearest-hit traversal and shading.  rayhierarchy
    // batches share the scene's status words, and a learned ordering that
    // serves nearest-hit batches shares its prediction and record buffers
    // with the any-hit ones, so those frames stay serial.
    const bool overlap = prm->integrator == PBG_INTEGRATOR_PATH &&
                         (s->accel == PBG_ACCEL_RAYBVH || s->accel == PBG_ACCEL_NAIVE) &&
                         !(s->learn && s->learn->enabled && (s->learn->queries & 1));
    // Queue lengths stay on the device where every walk of the frame can read
    // them there: the host then enqueues the bounces without waiting.
    const bool device_counts = !stream && s->accel == PBG_ACCEL_RAYBVH && bvh_queue_ok(s);
    if ((r = ensure(B.o4, n * 16)) || (r = ensure(B.d4, n * 16)) || (r = ensure(B.qidx[0], n * 4)) ||
        (r = ensure(B.qidx[1], n * 4)) || (r = ensure(B.qidx[2], n * 4)) ||
        (r = ensure(B.L, n * 12)) || (r = ensure(B.beta, n * 12)) || (r = ensure(B.prim, n * 4)) ||
        (r = ensure(B.t, n * 4)) || (r = ensure(B.b1, n * 4)) || (r = ensure(B.b2, n * 4)) ||
        (r = ensure(B.o42, n * 16)) || (r = ensure(B.d42, n * 16)) || (r = ensure(B.rgb, npix * 12)) ||
        (r = ensure(B.rstat, 16)) || (r = ensure(B.ltab, (size_t)std::max(ltab_floats, 1) * 4)) ||
        (r = ensure(B.bcount, kCountedBounces * sizeof(BounceCount))))
        return r;
    if (stream && ((r = ensure(B.no, n * 16)) || (r = ensure(B.nd, n * 16)) || (r = ensure(B.nflag, n)) ||
                   (r = ensure(B.counts, ((nk + 255) / 256 + 64) * 4 + 4096))))
        return r;
    for (int k = 0; k < (overlap ? 2 : 1); ++k) {
        ShadowSet& X = B.sh[k];
        if ((r = ensure(X.scontrib, nk * 12)) || (r = ensure(X.spos, nk * 4)) || (r = ensure(X.sqo, nk * 16)) ||
            (r = ensure(X.sqd, nk * 16)) || (r = ensure(X.occ, nk)) || (emitters && (r = ensure(X.emit, n * 12))))
            return r;
        if (stream && ((r = ensure(X.so, nk * 16)) || (r = ensure(X.sd, nk * 16)) || (r = ensure(X.sflag, nk)))) return r;
    }
    if (!B.words) PBG_CUDA(cudaHostAlloc((void**)&B.words, sizeof(RenderBuffers::HostWords), cudaHostAllocDefault));
    for (cudaEvent_t& e : B.span)
        if (!e) PBG_CUDA(cudaEventCreate(&e));
    // a frame that ended early on an error may have left work on the side stream
    if (B.side) PBG_CUDA(cudaStreamSynchronize(B.side));
    if (overlap && !B.side) {
        PBG_CUDA(cudaStreamCreateWithFlags(&B.side, cudaStreamNonBlocking));
        for (int k = 0; k < 2; ++k) {
            PBG_CUDA(cudaEventCreateWithFlags(&B.ready[k], cudaEventDisableTiming));
            PBG_CUDA(cudaEventCreateWithFlags(&B.resolved[k], cudaEventDisableTiming));
        }
    }
    PBG_CUDA(cudaMemsetAsync(B.rstat.ptr, 0, 16, st));
    rc.ltab = (const float*)B.ltab.ptr;
    for (int l = 0; l < nlights; ++l)
        if (rc.lights[l].type == PBG_LIGHT_MESH) {
            emitter_setup_kernel<<<1, 32, 0, st>>>((const float*)s->tri9.ptr, rc.lights[l].first, rc.lights[l].ntri,
                                                   (float*)B.ltab.ptr + rc.lights[l].tab);
            PBG_CUDA(cudaGetLastError());
            s->counters.kernel_launches += 1;
        }
    StreamArgs sa{};
    const int32_t* film_off = nullptr;
    const int32_t* film_idx = nullptr;
    if (stream) {
        // the caller's sample values, and each pixel's samples in order
        const size_t nd = (size_t)stream->ndims;
        std::vector<int32_t> cnt(npix + 1, 0);
        for (int64_t i = 0; i < n; ++i) {
            int x0, x1, y0, y1;
            film_footprint(stream->image_xy[2 * i], stream->image_xy[2 * i + 1], cam->xres, cam->yres, &x0, &x1, &y0, &y1);
            for (int y = y0; y <= y1; ++y)
                for (int x = x0; x <= x1; ++x) cnt[(int64_t)y * cam->xres + x + 1]++;
        }
        for (int64_t p = 0; p < npix; ++p) cnt[p + 1] += cnt[p];
        std::vector<int32_t> idx(std::max<int32_t>(cnt[npix], 1)), fill(cnt.begin(), cnt.end() - 1);
        for (int64_t i = 0; i < n; ++i) {
            int x0, x1, y0, y1;
            film_footprint(stream->image_xy[2 * i], stream->image_xy[2 * i + 1], cam->xres, cam->yres, &x0, &x1, &y0, &y1);
            for (int y = y0; y <= y1; ++y)
                for (int x = x0; x <= x1; ++x) idx[fill[(int64_t)y * cam->xres + x]++] = (int32_t)i;
        }
        if ((r = ensure(B.simg, n * 8)) || (r = ensure(B.sdims, n * nd * 4)) ||
            (r = ensure(B.srng, (size_t)std::max<int64_t>(stream->nrng, 1) * 4)) || (r = ensure(B.hflag, n)) ||
            (r = ensure(B.hrank, n * 4)) || (r = ensure(B.foff, (npix + 1) * 4)) ||
            (r = ensure(B.fidx, idx.size() * 4)))
            return r;
        PBG_CUDA(cudaMemcpyAsync(B.simg.ptr, stream->image_xy, n * 8, cudaMemcpyHostToDevice, st));
        PBG_CUDA(cudaMemcpyAsync(B.sdims.ptr, stream->dims, n * nd * 4, cudaMemcpyHostToDevice, st));
        if (stream->nrng > 0)
            PBG_CUDA(cudaMemcpyAsync(B.srng.ptr, stream->rng, stream->nrng * 4, cudaMemcpyHostToDevice, st));
        PBG_CUDA(cudaMemcpyAsync(B.foff.ptr, cnt.data(), (npix + 1) * 4, cudaMemcpyHostToDevice, st));
        PBG_CUDA(cudaMemcpyAsync(B.fidx.ptr, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice, st));
        PBG_CUDA(cudaStreamSynchronize(st));  // the host vectors go out of scope
        sa.img = (const float*)B.simg.ptr;
        sa.dims = (const float*)B.sdims.ptr;
        sa.rng = (const float*)B.srng.ptr;
        sa.count = n;
        sa.nrng = stream->nrng;
        sa.ndims = stream->ndims;
        film_off = (const int32_t*)B.foff.ptr;
        film_idx = (const int32_t*)B.fidx.ptr;
    }
    PBG_CUDA(cudaEventRecord(B.span[0], st));
    raygen_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        rc, sa, n, (float4*)B.o4.ptr, (float4*)B.d4.ptr, (int32_t*)B.qidx[0].ptr, (float*)B.L.ptr,
        (float*)B.beta.ptr);
    PBG_CUDA(cudaGetLastError());
    s->counters.kernel_launches += 1;
    pbg_render_stats stt{};
    stt.camera_rays = (uint64_t)n;
    int64_t nq = n;
    int64_t rng_base = 0;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    // Ray arrays alternate; queue indices rotate over three, since a bounce's
    // resolve reads its own while the next bounce's shade already fills the
    // one after the next.
    float4 *qo = (float4*)B.o4.ptr, *qd = (float4*)B.d4.ptr, *qo2 = (float4*)B.o42.ptr, *qd2 = (float4*)B.d42.ptr;
    BounceCount* counts = (BounceCount*)B.bcount.ptr;
    // camera rays and their shadow rays are coherent, later bounces are not
    struct HintGuard {
        pbg_scene* s;
        int32_t samples;
        ~HintGuard() {
            s->walk_hint = -1;
            s->samples = samples;
        }
    } hint_guard{s, s->samples};
    s->samples = stream ? 0 : rc.spp;
    cudaStream_t side = overlap ? B.side : st;
    bool pending[2] = {false, false};  // a resolve on the side stream still reads set k
    const uint32_t* nq_dev = nullptr;  // the queue's length on the device (nq: its upper bound)
    // grid-stride kernels over a queue of unknown length: 16 CTAs of 128 threads per SM
    auto grid_of = [&](int64_t items, int threads) {
        const int64_t blocks = (items + threads - 1) / threads;
        return (unsigned)(nq_dev ? std::min<int64_t>(blocks, (int64_t)sms * 16 * 128 / threads) : blocks);
    };
    // the counts of the bounces since the last reset, once they are complete
    auto add_counts = [&](int bounces) {
        for (int b = 0; b < bounces; ++b) {
            const BounceCount& c = B.words->count[b];
            if (c.nshadow > 0) s->counters.calls++;
            s->counters.rays_occluded += c.nshadow;
            stt.shadow_rays += c.nshadow;
            if (c.nnext > 0 && b + 1 < bounces) s->counters.calls++;
            if (b + 1 < bounces) {  // bounce b + 1 of this run traced them
                s->counters.rays_nearest += c.nnext;
                stt.nearest_rays += c.nnext;
                if (c.nnext > 0) stt.bounces++;
            }
        }
    };
    int counted = 0;  // bounces enqueued since the last reset
    for (int bounce = 0; nq > 0; ++bounce) {
        s->walk_hint = bounce > 0 ? 1 : 0;
        const int k = overlap ? (bounce & 1) : 0;
        ShadowSet& X = B.sh[k];
        const int32_t* qi = (const int32_t*)B.qidx[bounce % 3].ptr;
        int32_t* qi2 = (int32_t*)B.qidx[(bounce + 1) % 3].ptr;
        if (bounce % kCountedBounces == 0) {
            if (bounce > 0 && device_counts) {  // all bounces so far have ended (below)
                add_counts(counted);
                counted = 0;
                nq_dev = nullptr;
                nq = B.words->count[kCountedBounces - 1].nnext;
                if (nq == 0) break;
            }
            counted = 0;
            PBG_CUDA(cudaMemsetAsync(counts, 0, kCountedBounces * sizeof(BounceCount), st));
        }
        BounceCount* C = counts + bounce % kCountedBounces;
        if (nq_dev) {
            if ((r = bvh_queue_nearest(s, qo, qd, nq, nq_dev, &C->next_near, (int32_t*)B.prim.ptr, (float*)B.t.ptr,
                                       (float*)B.b1.ptr, (float*)B.b2.ptr, st)))
                return r;
        } else {
            if ((r = pbg_intersect_device(s, (const float*)qo, (const float*)qd, nullptr, nq,
                                          (int32_t*)B.prim.ptr, (float*)B.t.ptr, (float*)B.b1.ptr,
                                          (float*)B.b2.ptr, st)))
                return r;
            stt.nearest_rays += (uint64_t)nq;
            if (rc.integrator == PBG_INTEGRATOR_PATH) stt.bounces++;
        }
        const bool draws = stream && rc.integrator == PBG_INTEGRATOR_PATH && bounce >= 3;
        int64_t nhits = 0;
        if (draws) {
            hit_flag_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>((const int32_t*)B.prim.ptr, nq,
                                                                           (uint8_t*)B.hflag.ptr);
            PBG_CUDA(cudaGetLastError());
            s->counters.kernel_launches += 1;
            if ((r = compact_count(s, (const uint8_t*)B.hflag.ptr, nq, (uint32_t*)B.counts.ptr, &nhits, st))) return r;
            hit_rank_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(
                (const uint8_t*)B.hflag.ptr, nq, (const uint32_t*)B.counts.ptr, (int32_t*)B.hrank.ptr);
            PBG_CUDA(cudaGetLastError());
            s->counters.kernel_launches += 1;
            if (rng_base + 7 * n + nhits * (bounce > 3 ? 4 : 3) > stream->nrng) {
                set_last_error("pbg_render_stream: the stream's RNG draws ran out");
                return PBG_ERR_INVALID_ARGUMENT;
            }
            sa.rng_base = rng_base;
            sa.hit_rank = (const int32_t*)B.hrank.ptr;
        }
        const int64_t nslots = nq * kslots;
        // set k, and the queue that this bounce's shade fills, were last read
        // by the resolve of two bounces ago
        if (pending[k]) PBG_CUDA(cudaStreamWaitEvent(st, B.resolved[k], 0));
        pending[k] = false;
        ShadeIO io{};
        io.nq = nq;
        io.nq_dev = nq_dev;
        io.qidx = qi;
        io.qo = qo;
        io.qd = qd;
        io.prim = (const int32_t*)B.prim.ptr;
        io.th = (const float*)B.t.ptr;
        io.b1 = (const float*)B.b1.ptr;
        io.b2 = (const float*)B.b2.ptr;
        io.so = (float4*)(stream ? X.so.ptr : X.sqo.ptr);
        io.sd = (float4*)(stream ? X.sd.ptr : X.sqd.ptr);
        io.spos = (int32_t*)X.spos.ptr;
        io.nshadow = &C->nshadow;
        io.nidx = qi2;
        io.no = stream ? (float4*)B.no.ptr : qo2;
        io.nd = stream ? (float4*)B.nd.ptr : qd2;
        io.nnext = &C->nnext;
        io.sflag = (uint8_t*)X.sflag.ptr;
        io.nflag = (uint8_t*)B.nflag.ptr;
        io.scontrib = (float*)X.scontrib.ptr;
        io.emit = emitters && bounce == 0 ? (float*)X.emit.ptr : nullptr;
        const bool direct = rc.integrator == PBG_INTEGRATOR_DIRECT;
        auto shade = stream ? (direct ? shade_kernel<true, true> : shade_kernel<true, false>)
                            : (direct ? shade_kernel<false, true> : shade_kernel<false, false>);
        shade<<<grid_of(nq, kShadeThreads), kShadeThreads, 0, st>>>(
            rc, sa, bounce, io, (const float*)s->tri9.ptr, (const float*)s->uv6.ptr, (float*)B.beta.ptr, kslots,
            (int*)B.rstat.ptr);
        PBG_CUDA(cudaGetLastError());
        s->counters.kernel_launches += 1;
        if (draws) rng_base += 7 * n + nhits * (bounce > 3 ? 4 : 3);
        int64_t nsh = 0, nn = 0;
        if (stream) {  // the slots and the bounce rays in order
            if ((r = compact_count(s, (const uint8_t*)X.sflag.ptr, nslots, (uint32_t*)B.counts.ptr, &nsh, st)))
                return r;
            compact_shadow_kernel<<<(unsigned)((nslots + 255) / 256), 256, 0, st>>>(
                (const uint8_t*)X.sflag.ptr, nslots, (const uint32_t*)B.counts.ptr, (const float4*)X.so.ptr,
                (const float4*)X.sd.ptr, (float4*)X.sqo.ptr, (float4*)X.sqd.ptr, (int32_t*)X.spos.ptr);
            PBG_CUDA(cudaGetLastError());
            s->counters.kernel_launches += 1;
        } else if (!device_counts) {
            int h[2] = {0, 0};
            if ((r = read_device_words(s, (const int*)C, 2, h, st))) return r;
            nsh = h[0];
            nn = h[1];
        }
        if (overlap) {  // the shadow rays and this bounce's resolve on the side stream
            PBG_CUDA(cudaEventRecord(B.ready[k], st));
            PBG_CUDA(cudaStreamWaitEvent(side, B.ready[k], 0));
        }
        if (device_counts) {
            if ((r = bvh_queue_occluded(s, (const float4*)X.sqo.ptr, (const float4*)X.sqd.ptr, nslots, &C->nshadow,
                                        &C->next_any, (uint8_t*)X.occ.ptr, side)))
                return r;
        } else if (nsh > 0) {
            if (overlap) std::swap(s->work, s->alt);  // its own walk counter, beside the nearest-hit walk
            r = pbg_occluded_device(s, (const float*)X.sqo.ptr, (const float*)X.sqd.ptr, nullptr, nsh,
                                    (uint8_t*)X.occ.ptr, side);
            if (overlap) std::swap(s->work, s->alt);
            if (r) return r;
        }
        stt.shadow_rays += (uint64_t)nsh;
        resolve_kernel<<<grid_of(nq, 256), 256, 0, side>>>(
            rc, nq, nq_dev, kslots, qi, (const int32_t*)X.spos.ptr, (const uint8_t*)X.occ.ptr,
            (const float*)X.scontrib.ptr, io.emit, (float*)B.L.ptr);
        PBG_CUDA(cudaGetLastError());
        s->counters.kernel_launches += 1;
        if (overlap) {
            PBG_CUDA(cudaEventRecord(B.resolved[k], side));
            pending[k] = true;
        }
        ++counted;
        if (rc.integrator != PBG_INTEGRATOR_PATH) break;
        if (stream) {
            if ((r = compact_count(s, (const uint8_t*)B.nflag.ptr, nq, (uint32_t*)B.counts.ptr, &nn, st)))
                return r;
            compact_bounce_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(
                (const uint8_t*)B.nflag.ptr, nq, (const uint32_t*)B.counts.ptr, qi, (const float4*)B.no.ptr,
                (const float4*)B.nd.ptr, qi2, qo2, qd2);
            PBG_CUDA(cudaGetLastError());
            s->counters.kernel_launches += 1;
        }
        std::swap(qo, qo2);
        std::swap(qd, qd2);
        if (!device_counts) {
            nq = nn;
            continue;
        }
        if (bounce >= rc.max_depth) break;  // no path goes on
        nq_dev = &C->nnext;
        if ((bounce + 1) % kCountedBounces == 0) {  // read the counts and wait, so that the next bounces can reuse them
            for (int q = 0; q < 2; ++q)
                if (pending[q]) PBG_CUDA(cudaStreamWaitEvent(st, B.resolved[q], 0));
            pending[0] = pending[1] = false;
            PBG_CUDA(cudaMemcpyAsync(B.words->count, counts, kCountedBounces * sizeof(BounceCount),
                                     cudaMemcpyDeviceToHost, st));
            PBG_CUDA(cudaStreamSynchronize(st));
        }
    }
    for (int k = 0; k < 2; ++k)  // the last resolves add to L before the film reads it
        if (pending[k]) PBG_CUDA(cudaStreamWaitEvent(st, B.resolved[k], 0));
    // online training of the learned ordering on this frame's records
    if (s->learn && s->learn->enabled && (r = learn_train(s, 0, st))) return r;
    film_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(npix, rc.spp, film_off, film_idx,
                                                                 (const float*)B.L.ptr, (float*)B.rgb.ptr);
    PBG_CUDA(cudaGetLastError());
    s->counters.kernel_launches += 1;
    PBG_CUDA(cudaEventRecord(B.span[1], st));
    RenderBuffers::HostWords& W = *B.words;
    if (device_counts)
        PBG_CUDA(cudaMemcpyAsync(W.count, counts, sizeof(W.count), cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaMemcpyAsync(W.rstat, B.rstat.ptr, 16, cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaMemcpyAsync(W.status, s->err.ptr, 16, cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaMemcpyAsync(rgb_host, B.rgb.ptr, npix * 12, cudaMemcpyDeviceToHost, st));
    PBG_CUDA(cudaStreamSynchronize(st));
    if (device_counts) add_counts(counted);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, B.span[0], B.span[1]);
    stt.ms_total = ms;
    if (stats) *stats = stt;
    const int* rstat = W.rstat;
    if (rstat[0] != 0) {
        char buf[200];
        snprintf(buf, sizeof(buf),
                 "pbg_render_stream: %d path vertices sampled a direction the BSDF rejects; the reference traces "
                 "such a ray again unchanged, so the stream no longer matches it",
                 rstat[0]);
        set_last_error(buf);
        return PBG_ERR_UNSUPPORTED;
    }
    if (W.status[kStatusTimeout] == 0 && W.status[kStatusOverflow] == 0) return PBG_OK;
    return check_device_status(s, st);  // reports and clears them
}

}  // namespace pbg

extern "C" int pbg_render(pbg_scene* scene, const pbg_camera* camera, const pbg_light* lights,
                          int32_t nlights, const pbg_render_params* params, float* rgb,
                          pbg_render_stats* stats) {
    if (!scene) {
        pbg::set_last_error("pbg_render: scene is NULL");
        return PBG_ERR_INVALID_ARGUMENT;
    }
    cudaSetDevice(scene->device);
    return pbg::render(scene, camera, lights, nlights, params, nullptr, rgb, stats);
}

extern "C" int pbg_render_stream(pbg_scene* scene, const pbg_camera* camera, const pbg_light* lights,
                                 int32_t nlights, const pbg_render_params* params,
                                 const pbg_sample_stream* stream, float* rgb, pbg_render_stats* stats) {
    if (!scene || !stream) {
        pbg::set_last_error("pbg_render_stream: scene or stream is NULL");
        return PBG_ERR_INVALID_ARGUMENT;
    }
    cudaSetDevice(scene->device);
    return pbg::render(scene, camera, lights, nlights, params, stream, rgb, stats);
}
