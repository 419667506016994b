// pbg_wide.cuh -- the walk over an eight-wide BVH (ray-bvh walks 5 and 6,
// and the scene set's wide walks), templated on where its rays come from.
//
// Src supplies: count() rays; fetch(slot, lane, o, d) -> false for a ray
// that is not traced (a miss); nodes / tris / unculled of a lane's scene;
// store<ANY>(lane, hit); kSet with scene(lane) and stamp(scene) for a scene
// set's completion stamps.  The node layout and the walk are described in
// pbg_wide.cu.
#pragma once
#include <vector>

#include "pbg_internal.h"
#ifdef __CUDACC__
#include "pbg_tma.cuh"
#include "pbg_walk.cuh"
#endif

namespace pbg {

struct __align__(16) WideNode {
    float4 plane[12];  // per axis: lo[0-3], lo[4-7], hi[0-3], hi[4-7]
    int4 refs;         // child_base | imask << 24, tri_base, 0, 0
    uint4 tris[2];     // per slot: its leaf's triangles as bits of the node's triangle mask (0: inner or empty)
};
static_assert(sizeof(WideNode) == 240, "wide node is fifteen 16-byte words");

// The collapse of a binary tree (pbg_wide.cu); false when the tree does not
// fit the wide format.
bool collapse_wide(const std::vector<BvhNode>& bin, int32_t unculled, int64_t ntri, int absorb, float c_tri,
                   std::vector<WideNode>* out, std::vector<int32_t>* src);
constexpr int kWideWidth = 8;         // children per node
constexpr int kWideMaxLeaf = 7;       // triangles per leaf child
constexpr int kWideMaxOffset = 31;    // a leaf's first triangle within its node's 32
constexpr int kWideAbsorb = 4;        // subtrees of at most this many triangles may become one leaf
constexpr float kWideTriCost = 0.3f;  // a triangle test against a wide node visit

#ifdef __CUDACC__
constexpr int kWideThreads = 128;
constexpr int kWideMinBlocks = 7;  // CTAs per SM: 7 measured best of 5, 6, 7, 8
constexpr int kWideStack = 64;

// A group's entry distance kept in the upper 16 bits of a stack word,
// rounded toward -infinity (a popped group is skipped only when it lies
// beyond the hit found).
__device__ __forceinline__ uint32_t dist_bits_down(float t) {
    uint32_t b = __float_as_uint(t);
    if (b & 0x80000000u) b += 0xffffu;  // negative: a larger magnitude is smaller
    return b & 0xffff0000u;
}

// COOP (walk 6): the triangle tests of a warp's lanes spread over all 32
// lanes: lane j of round r tests pending pair r * 32 + j (pairs numbered
// lane by lane) against its owner's ray, read from shared memory; hits merge
// per owner by a 64-bit atomic maximum of hit_key (nearer t, then the larger
// index: the rule of pbrt's in-order loop that the other kernels keep too).
// It pays on incoherent batches, where a lane's pending triangles range from
// 1 to 64 (path bounces: nearest hit 1.77 -> 1.65 ms); on coherent ones the
// lanes' counts are alike and the shared-memory round trip costs more
// (camera rays 3.29 -> 4.15 ms), so the autotuner picks per batch class.

struct CoopWarp {
    float4 o[32], d[32];
    const TriRec* tris[32];      // the owner's records (scene sets)
    unsigned long long key[32];  // nearest: best hit_key (0: none); any-hit: nonzero once occluded
    float ht[32], nd[32], t[32], b1[32], b2[32];
    uint32_t m1[32], m2[32], m3[32];
    int32_t base1[32], base2[32], base3[32], off[32], occluder[32];
    int2 queue[64];              // (owner, record) for the exact test
};

// Children in visiting order: slot ^ visit_order(octant).  Nearest hits go
// front to back; any-hit rays back to front: a shadow ray's first boxes front
// to back are the surface around its origin, which it leaves, and its
// occluders lie farther on (path frame: shadow batches 0.70 -> 0.59 ms,
// camera shadows 3.89 -> 3.50 ms).
template <bool ANY>
__device__ __forceinline__ uint32_t visit_order_of(uint32_t oct) { return ANY ? oct ^ 7u : oct; }

template <bool ANY, bool STATS, bool COOP, class Src>
__global__ void __launch_bounds__(kWideThreads, kWideMinBlocks)
    wide_walk_kernel(const Src src, int* status, unsigned long long* next, unsigned long long* wcount) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ CoopWarp coop[COOP ? kWideThreads / 32 : 1];
    // eight hit bits in visiting order: bit k to bit k ^ order (a table: the
    // three conditional swaps took 15 instructions a visit), made four entries
    // to a word
    __shared__ __align__(4) uint8_t visit[8][256];
    for (int i = threadIdx.x; i < 8 * 64; i += kWideThreads) {
        const uint32_t vo = (uint32_t)i >> 6;
        uint32_t m = ((uint32_t)i & 63u) * 0x04040404u + 0x03020100u;
        if (vo & 1u) m = ((m & 0x55555555u) << 1) | ((m >> 1) & 0x55555555u);
        if (vo & 2u) m = ((m & 0x33333333u) << 2) | ((m >> 2) & 0x33333333u);
        if (vo & 4u) m = ((m & 0x0f0f0f0fu) << 4) | ((m >> 4) & 0x0f0f0f0fu);
        reinterpret_cast<uint32_t*>(visit)[i] = m;
    }
    __syncthreads();
    int2 stack[kWideStack];  // (child base, hits | imask << 8 | distance bits)
    int sp = 0;
    typename Src::Lane L{};
    bool has = false, exhausted = false, ok = true, fin = false;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
    RayFma rf{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float nd = 0.f;
    WalkHit h{0.f, 0.f, 0.f, -1};
    uint32_t oct = 0;
    int32_t gbase = 0;          // the current group: inner children from gbase
    uint32_t ghits = 0, gimask = 0;  // hit children in visiting order, the node's inner mask
    float gtn = 0.f;            // the group's nearest entry distance
    int32_t tbase = 0;          // pending triangles of the last node: records tbase + bit
    uint32_t tmask = 0;
    int32_t tbase2 = 0;         // a second node's triangles, found while others searched
    uint32_t tmask2 = 0;
    int32_t tbase3 = 0;         // walk 6: a third (its tests are dealt over the warp)
    uint32_t tmask3 = 0;
    int32_t rcnt = 0;           // pending degenerate records [0, rcnt)
    WorkCount wc;

    auto finish = [&]() {
        src.template store<ANY>(L, h);
        if (!ok) atomicAdd(&status[kStatusOverflow], 1);
        has = false;
        fin = true;
    };

    const int64_t n = src.count();
    for (;;) {
        fin = false;
        // refill the lanes whose ray is done
        const unsigned need = __ballot_sync(full, !has && !exhausted);
        if (need) {
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(next, (unsigned long long)__popc(need));
            base = __shfl_sync(full, base, leader);
            if (!has && !exhausted) {
                const int64_t slot = (int64_t)base + __popc(need & lt);
                if (slot >= n) {
                    exhausted = true;
                } else {
                    if (!src.fetch(slot, L, o, d)) {
                        h = WalkHit{0.f, 0.f, 0.f, -1};
                        ok = true;
                        finish();  // invalid: a miss, no walk
                    } else {
                        nd = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
                        rf = ray_fma(o, d);
                        oct = (__float_as_uint(rf.ix) >> 31) | (__float_as_uint(rf.iy) >> 31) << 1 |
                              (__float_as_uint(rf.iz) >> 31) << 2;
                        h = unhit(d);
                        sp = 0;
                        ok = true;
                        gbase = 0;  // the root: slot 0 of a group whose only inner child is node 0
                        gimask = 1u;
                        ghits = 1u << visit_order_of<ANY>(oct);
                        gtn = -INFINITY;
                        tmask = 0;
                        tmask2 = 0;
                        tmask3 = 0;
                        rcnt = src.unculled(L);  // degenerate records first
                        has = true;
                    }
                }
            }
        }
        if (!__any_sync(full, has)) {
            if (__all_sync(full, exhausted)) break;
            continue;
        }
        // nodes until every lane holds triangles or has ended its ray
        for (;;) {
            const bool searching = has && tmask == 0 && rcnt == 0;
            if (!__any_sync(full, searching)) break;
            // walk 6: the tests are dealt over the warp, so they need not
            // wait for the last searching lane: once six lanes hold two
            // nodes' triangles the warp tests (64 scenes 5.28 / 5.21 / 5.16 /
            // 5.15 / 5.16 ms and path frame 17.6 / 17.5 / 17.4 / 17.5 / 17.7 ms
            // for 3, 4, 6, 8 and 12 such lanes)
            if (COOP && __popc(__ballot_sync(full, has && tmask2 != 0)) >= 6) break;
            // any-hit rays end at very different times: with 16 lanes idle
            // the warp takes new rays (direct lighting 966 -> 933 us; for
            // nearest hits 18.87 -> 19.12 ms, so not there)
            if (ANY && __popc(__ballot_sync(full, !has && !exhausted)) >= 16) break;
            // a lane that holds triangles walks on for one more node's
            // triangles (two more when the warp deals its tests over its
            // lanes) while others search, so the tests below run with fuller
            // warps (walk 6 with two more: path bounces 1.66 -> 1.64 ms)
            const bool act = has && !(COOP ? tmask3 != 0 : tmask2 != 0) && rcnt == 0;
            // A lane out of children takes its next group here and visits it
            // in the same step.  The barrier brings the warp back together:
            // without it the compiler ran the visit once for the lanes that
            // popped and once for the others (path frame 21.2 -> 23.3 ms; with
            // it 19.6 -> 19.1 over popping in a step of its own).
            if (act) {
                if (ghits != 0 && gtn > h.t) ghits = 0;  // the whole group lies beyond the hit found
                while (ghits == 0 && sp > 0) {
                    --sp;
                    const int2 e = stack[sp];
                    const float te = __uint_as_float((uint32_t)e.y & 0xffff0000u);
                    if (!(te > h.t)) {
                        gbase = e.x;
                        ghits = (uint32_t)e.y & 0xffu;
                        gimask = ((uint32_t)e.y >> 8) & 0xffu;
                        gtn = te;
                    }
                }
            }
            __syncwarp();
            if (!act) continue;
            if (ghits == 0) {
                if (tmask == 0) finish();  // nothing left to walk or test
                continue;
            }
            const int pos = __ffs(ghits) - 1;
            const uint32_t rest = ghits & (ghits - 1u);
            const int cslot = pos ^ (int)visit_order_of<ANY>(oct);
            const int32_t child = gbase + __popc(gimask & ((1u << cslot) - 1u));

            // 32-bit offsets from the tree's base (under 2^24 nodes): fewer
            // address instructions than a 64-bit pointer per plane
            const char* nb = reinterpret_cast<const char*>(src.nodes(L));
            const uint32_t at = (uint32_t)child * (uint32_t)sizeof(WideNode);
            auto ld = [&](uint32_t word) { return __ldg(reinterpret_cast<const float4*>(nb + (at + word * 16u))); };
            const int4 r = __ldg(reinterpret_cast<const int4*>(nb + (at + 192u)));
            const uint32_t xo = (oct & 1u) * 2u, yo = 4u + (oct & 2u), zo = 8u + (oct & 4u) / 2u;
            const float4 nx0 = ld(xo), nx1 = ld(xo + 1u), fx0 = ld(2u - xo), fx1 = ld(3u - xo);
            const float4 ny0 = ld(yo), ny1 = ld(yo + 1u), fy0 = ld(10u - yo), fy1 = ld(11u - yo);
            const float4 nz0 = ld(zo), nz1 = ld(zo + 1u), fz0 = ld(18u - zo), fz1 = ld(19u - zo);
            const uint4 lt0 = __ldg(reinterpret_cast<const uint4*>(nb + (at + 208u)));
            const uint4 lt1 = __ldg(reinterpret_cast<const uint4*>(nb + (at + 224u)));
            const uint32_t lts[8] = {lt0.x, lt0.y, lt0.z, lt0.w, lt1.x, lt1.y, lt1.z, lt1.w};
            const uint32_t imask = (uint32_t)r.x >> 24;
            uint32_t hits = 0, tm = 0;
            float ntn = INFINITY;  // nearest entry over the hit children: a bound for the group
            const float2 ix2 = make_float2(rf.ix, rf.ix), iy2 = make_float2(rf.iy, rf.iy), iz2 = make_float2(rf.iz, rf.iz);
            const float2 cx2 = make_float2(rf.cx, rf.cx), cy2 = make_float2(rf.cy, rf.cy), cz2 = make_float2(rf.cz, rf.cz);
            const float4 nxs[2] = {nx0, nx1}, fxs[2] = {fx0, fx1}, nys[2] = {ny0, ny1}, fys[2] = {fy0, fy1},
                         nzs[2] = {nz0, nz1}, fzs[2] = {fz0, fz1};
#pragma unroll
            for (int k = 0; k < kWideWidth; k += 2) {  // two boxes at a time
                const float2 tnx = fma2(pair_of(nxs, k), ix2, cx2), tfx = fma2(pair_of(fxs, k), ix2, cx2);
                const float2 tny = fma2(pair_of(nys, k), iy2, cy2), tfy = fma2(pair_of(fys, k), iy2, cy2);
                const float2 tnz = fma2(pair_of(nzs, k), iz2, cz2), tfz = fma2(pair_of(fzs, k), iz2, cz2);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float tn = fmax3(q ? tnx.y : tnx.x, q ? tny.y : tny.x, fmaxf(q ? tnz.y : tnz.x, o.w));
                    const float tf = fmin3(q ? tfx.y : tfx.x, q ? tfy.y : tfy.x, fminf(q ? tfz.y : tfz.x, h.t));
                    if (tn <= fmaf(fabsf(tf), kSlabWiden, tf)) {
                        hits |= 1u << (k + q);
                        tm |= lts[k + q];
                        if (!ANY) ntn = fminf(ntn, tn);
                    }
                }
            }
            if (STATS) {
                uint32_t occupied = imask;
#pragma unroll
                for (int k = 0; k < kWideWidth; ++k) occupied |= lts[k] != 0u ? 1u << k : 0u;
                wc.node += __popc(occupied);
            }
            // hit inner children in visiting order: bit (slot ^ octant)
            uint32_t ih = hits & imask;
            const uint32_t vo = visit_order_of<ANY>(oct);
            ih = visit[vo][ih];
            if (ih) {
                if (rest) {
                    if (sp < kWideStack) {
                        stack[sp] = make_int2(gbase, (int)(rest | gimask << 8 | dist_bits_down(gtn)));
                        ++sp;
                    } else {
                        ok = false;
                    }
                }
                gbase = r.x & 0xffffff;
                ghits = ih;
                gimask = imask;
                gtn = ANY ? -INFINITY : ntn;
            } else {
                ghits = rest;
            }
            if (tmask == 0) {
                tbase = r.y;
                tmask = tm;
            } else if (tmask2 == 0) {
                tbase2 = r.y;
                tmask2 = tm;
            } else {
                tbase3 = r.y;
                tmask3 = tm;
            }
        }
        // the triangle tests, converged
        if (COOP) {
            // degenerate records (a ray's first round only), one lane each
            if (has && rcnt != 0) {
                const bool done = test_run<ANY, STATS>(src.tris(L), 0, rcnt, o, d, nd, h, wc);
                rcnt = 0;
                if (done) {
                    tmask = tmask2 = tmask3 = 0;
                    finish();
                }
            }
            const bool mine = has && (tmask | tmask2 | tmask3) != 0;
            const int c = mine ? __popc(tmask) + __popc(tmask2) + __popc(tmask3) : 0;
            int incl = c;
#pragma unroll
            for (int sh = 1; sh < 32; sh <<= 1) {
                const int v = __shfl_up_sync(full, incl, sh);
                if (lane >= sh) incl += v;
            }
            const int total = __shfl_sync(full, incl, 31);
            if (total > 0) {
                CoopWarp& cw = coop[threadIdx.x >> 5];
                const unsigned long long own = ANY || h.prim < 0 ? 0ull : hit_key(h.t, h.prim);
                cw.off[lane] = incl - c;
                if (mine) {
                    if (STATS) wc.leaf++;
                    cw.o[lane] = o;
                    cw.d[lane] = d;
                    if (Src::kSet) cw.tris[lane] = src.tris(L);
                    cw.nd[lane] = nd;
                    cw.ht[lane] = h.t;
                    cw.m1[lane] = tmask;
                    cw.m2[lane] = tmask2;
                    cw.m3[lane] = tmask3;
                    cw.base3[lane] = tbase3;
                    cw.base1[lane] = tbase;
                    cw.base2[lane] = tbase2;
                    cw.key[lane] = own;
                }
                __syncwarp();
                // Pairs that pass the filter queue for the exact test, which
                // runs for 32 of them or after the last round: some four of a
                // round's 32 pass, and it takes as long for one as for 32
                // (path bounces 938 -> 788 us, path frame 18.9 -> 17.5 ms, 64
                // scenes 5.93 -> 5.19 ms).
                int queued = 0;
                for (int g0 = 0; g0 < total || queued > 0; g0 += 32) {
                    const int g = g0 + lane;
                    bool cand = false;
                    int i = 0;  // the owner: the last lane whose first pair is <= g
                    int32_t rec = 0;
                    if (g < total) {
#pragma unroll
                        for (int step = 16; step; step >>= 1)
                            if (cw.off[i + step] <= g) i += step;
                        const int k = g - cw.off[i];
                        const uint32_t m1 = cw.m1[i];
                        const int n1 = __popc(m1);
                        const uint32_t m2v = cw.m2[i];
                        const int n2 = __popc(m2v);
                        rec = k < n1        ? cw.base1[i] + (int)__fns(m1, 0, k + 1)
                              : k < n1 + n2 ? cw.base2[i] + (int)__fns(m2v, 0, k - n1 + 1)
                                            : cw.base3[i] + (int)__fns(cw.m3[i], 0, k - n1 - n2 + 1);
                        if (!ANY || cw.key[i] == 0ull) {
                            if (STATS) wc.filt++;
                            cand = pbg_filter((Src::kSet ? cw.tris[i] : src.tris(L))[rec], cw.o[i], cw.d[i], cw.nd[i],
                                              cw.ht[i], STATS ? &wc.filt2 : nullptr);
                        }
                    }
                    const unsigned cm = __ballot_sync(full, cand);
                    if (cand) cw.queue[queued + __popc(cm & lt)] = make_int2(i, rec);
                    queued += __popc(cm);
                    if (queued == 0 || (queued < 32 && g0 + 32 < total)) continue;
                    __syncwarp();
                    const int take = min(queued, 32);
                    unsigned long long ck = 0ull;
                    float ct = 0.f, cu1 = 0.f, cu2 = 0.f;
                    int ci = -1;
                    if (lane < take) {
                        const int2 e = cw.queue[lane];
                        if (!ANY || cw.key[e.x] == 0ull) {
                            const TriRec tr = (Src::kSet ? cw.tris[e.x] : src.tris(L))[e.y];
                            if (STATS) wc.exact++;
                            if (pbg_exact_rec(tr, cw.o[e.x], cw.d[e.x], cw.ht[e.x], &ct, &cu1, &cu2)) {
                                if (STATS) wc.hit++;
                                const int32_t id = __float_as_int(tr.c.w);
                                if (ANY) {
                                    cw.key[e.x] = 1ull;
                                    cw.occluder[e.x] = id;
                                } else {
                                    ci = e.x;
                                    ck = hit_key(ct, id);
                                    atomicMax(&cw.key[ci], ck);
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (!ANY && ci >= 0 && cw.key[ci] == ck) {  // this round's winner for its owner
                        cw.t[ci] = ct;
                        cw.b1[ci] = cu1;
                        cw.b2[ci] = cu2;
                    }
                    int2 behind = make_int2(0, 0);
                    queued -= take;
                    if (lane < queued) behind = cw.queue[32 + lane];
                    __syncwarp();
                    if (lane < queued) cw.queue[lane] = behind;
                    __syncwarp();
                }
                if (mine) {
                    const unsigned long long kk = cw.key[lane];
                    if (ANY) {
                        if (kk != 0ull) {
                            h.prim = cw.occluder[lane];
                            finish();
                        }
                    } else if (kk != own) {
                        h.t = cw.t[lane];
                        h.prim = key_prim(kk);
                        h.b1 = cw.b1[lane];
                        h.b2 = cw.b2[lane];
                    }
                }
                __syncwarp();
            }
            tmask = 0;
            tmask2 = 0;
            tmask3 = 0;
        } else {
            const bool mine = has && (tmask != 0 || tmask2 != 0 || rcnt != 0);
            if (STATS && mine) wc.leaf++;
            bool done = false;
            if (mine && rcnt) {
                done = test_run<ANY, STATS>(src.tris(L), 0, rcnt, o, d, nd, h, wc);
                rcnt = 0;
            }
            // every lane on to its next record that passes the filter, then
            // the exact test for all of them together
            for (;;) {
                int32_t cand = -1;
                if (mine && !done) {
                    while (cand < 0 && (tmask | tmask2) != 0) {
                        const bool one = tmask != 0;
                        const uint32_t m = one ? tmask : tmask2;
                        const int32_t rec = (one ? tbase : tbase2) + __ffs(m) - 1;
                        if (one)
                            tmask = m & (m - 1u);
                        else
                            tmask2 = m & (m - 1u);
                        if (STATS) wc.filt++;
                        if (pbg_filter(src.tris(L)[rec], o, d, nd, h.t, STATS ? &wc.filt2 : nullptr)) cand = rec;
                    }
                }
                if (!__any_sync(full, cand >= 0)) break;
                if (cand >= 0) done = test_exact<ANY, STATS>(src.tris(L), cand, o, d, h, wc);
            }
            tmask = 0;
            tmask2 = 0;
            if (done) finish();
        }
        if (Src::kSet) {  // completion stamps: one atomic per scene per warp
            const int sc = fin ? src.scene(L) : -1;
            const unsigned m = __match_any_sync(full, sc);
            if (fin && lane == __ffs(m) - 1) src.stamp(sc);
        }
    }
    if (STATS) wc.flush(wcount);
}


// One scene's batch: the ray-bvh walks 5 and 6.
struct SceneRays {
    static constexpr bool kSet = false;
    struct Lane {
        int64_t ray;
    };
    const WideNode* wn;
    const TriRec* wt;
    int32_t unc;
    const float4* ro;
    const float4* rd;
    const uint8_t* valid;
    const int32_t* perm;
    int64_t n;
    const uint32_t* n_dev;  // the batch's length where the host does not know it
    int32_t* prim;
    float* t;
    float* b1;
    float* b2;
    uint8_t* occ;

    __device__ __forceinline__ int64_t count() const { return n_dev ? (int64_t)*n_dev : n; }
    __device__ __forceinline__ bool fetch(int64_t slot, Lane& L, float4& o, float4& d) const {
        L.ray = perm ? (int64_t)perm[slot] : slot;
        if (valid != nullptr && valid[L.ray] == 0) return false;
        o = ro[L.ray];
        d = rd[L.ray];
        return true;
    }
    __device__ __forceinline__ const WideNode* nodes(const Lane&) const { return wn; }
    __device__ __forceinline__ const TriRec* tris(const Lane&) const { return wt; }
    __device__ __forceinline__ int32_t unculled(const Lane&) const { return unc; }
    template <bool ANY>
    __device__ __forceinline__ void store(const Lane& L, const WalkHit& h) const {
        if (ANY) {
            occ[L.ray] = h.prim >= 0 ? 1 : 0;
            if (prim) prim[L.ray] = h.prim;
        } else {
            const bool hit = h.prim >= 0;
            prim[L.ray] = h.prim;
            t[L.ray] = hit ? h.t : 0.f;
            b1[L.ray] = hit ? h.b1 : 0.f;
            b2[L.ray] = hit ? h.b2 : 0.f;
        }
    }
    __device__ __forceinline__ int scene(const Lane&) const { return 0; }
    __device__ __forceinline__ void stamp(int) const {}
};
#endif  // __CUDACC__

}  // namespace pbg
