// pbg_rayorder.cu -- per-batch ray ordering: 6-D Morton keys and a
// hand-written LSD radix sort (warp-cooperative ranking).
//
// The reference arranges each batch as a 2-D ray image and groups rays by
// chunkX x chunkY image tiles (bin/cl/rayhconstruct6DB.cl:10-47,
// accelerators/rayhierarchy.cpp:375-463); that groups rays well only while
// they are camera rays in scanline order.  Here every batch -- camera,
// shadow or bounce rays -- is sorted by a 30-bit Morton code interleaving
// five bits each of origin x/y/z (quantised over the batch's origin box) and
// normalised direction x/y/z, so that consecutive rays share origin and
// direction whatever produced them.  Invalid rays get the key 0xffffffff and
// sort to the end.
//
// Sort (batches above 131,072 rays; smaller ones: sort_cluster_kernel, one
// launch): four passes of 8 bits.  Each pass is (1) a per-tile digit histogram,
// (2) one exclusive scan over [digit][tile] counts, (3) a stable scatter in
// which each warp ranks its 32 keys per digit with __match_any_sync and the
// tile's warps are combined through shared-memory prefix sums.
#include <algorithm>
#include <atomic>

#include "pbg_curve.cuh"
#include "pbg_internal.h"
#include "pbg_tma.cuh"

namespace pbg {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;                         // keys per thread
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys per tile
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kDigitBits = 8;  // 8 keys per digit per 2048-key tile keep the scatter coalesced
constexpr int kRadix = 1 << kDigitBits;
constexpr uint32_t kDigitMask = kRadix - 1;
// A sort of the low `bits` key bits: valid keys are clamped below
// 2^bits - 1, so an invalid ray's key 0xffffffff (low bits all ones) sorts
// after every valid one.
constexpr int kKeyBits = 30;                            // image and 6-D keys: 4 passes
constexpr int kOriginAxisBits = 8;  // origin keys: bits per axis (measured best of 5, 7, 8)
constexpr int kOriginKeyBits = 3 * kOriginAxisBits;     // 24 bits: 3 passes
constexpr uint32_t kMaxValidKey = (1u << kKeyBits) - 2u;
constexpr uint32_t kMaxOriginKey = (1u << kOriginKeyBits) - 2u;

__device__ __forceinline__ uint32_t spread5(uint32_t v) {
    // 5 bits -> positions 0, 6, 12, 18, 24
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b) r |= ((v >> b) & 1u) << (6 * b);
    return r;
}

__device__ __forceinline__ uint32_t quant5(float x, float lo, float inv_ext) {
    float q = (x - lo) * inv_ext * 32.f;
    q = fminf(fmaxf(q, 0.f), 31.f);
    return (uint32_t)q;
}

// Block-level min/max of valid ray origins (atomic on ordered ints).
__device__ __forceinline__ int ord_f(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float unord_f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void origin_bounds_kernel(const float4* __restrict__ ro, const uint8_t* __restrict__ valid,
                                     int64_t n, int* __restrict__ bounds /* lo xyz, hi xyz */) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (valid && !valid[i]) continue;
        const float4 o = ro[i];
        if (!(isfinite(o.x) && isfinite(o.y) && isfinite(o.z))) continue;
        lo[0] = fminf(lo[0], o.x); lo[1] = fminf(lo[1], o.y); lo[2] = fminf(lo[2], o.z);
        hi[0] = fmaxf(hi[0], o.x); hi[1] = fmaxf(hi[1], o.y); hi[2] = fmaxf(hi[2], o.z);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int off = 16; off; off >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; ++a) {
            atomicMin(&bounds[a], ord_f(lo[a]));
            atomicMax(&bounds[3 + a], ord_f(hi[a]));
        }
    }
}

// Empty bounds for origin_bounds_kernel's atomics: lo = max, hi = min.
__global__ void init_bounds_kernel(int* __restrict__ bounds) {
    if (threadIdx.x < 6) bounds[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : (int)0x80000000;
}

// The batch's origin box, from ordered integers.
struct OriginBox {
    float lo[3], hi[3];
};
__device__ __forceinline__ OriginBox origin_box(const int* b) {
    OriginBox r;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        r.lo[a] = unord_f(b[a]);
        r.hi[a] = unord_f(b[3 + a]);
    }
    return r;
}

__device__ __forceinline__ uint32_t morton_key(float4 o, float4 d, const OriginBox& box) {
    float inv[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float ext = box.hi[a] - box.lo[a];
        inv[a] = ext > 0.f ? 1.f / ext : 0.f;
    }
    const float len = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    const float il = len > 0.f ? 1.f / len : 0.f;
    uint32_t qo0 = quant5(o.x, box.lo[0], inv[0]), qo1 = quant5(o.y, box.lo[1], inv[1]),
             qo2 = quant5(o.z, box.lo[2], inv[2]);
    uint32_t qd0 = quant5(d.x * il, -1.f, 0.5f), qd1 = quant5(d.y * il, -1.f, 0.5f),
             qd2 = quant5(d.z * il, -1.f, 0.5f);
    // Direction bits above origin bits at each level: coherent directions first.
    return min(kMaxValidKey, (spread5(qd0) << 5) | (spread5(qd1) << 4) | (spread5(qd2) << 3) |
                                 (spread5(qo0) << 2) | (spread5(qo1) << 1) | spread5(qo2));
}

__global__ void morton_kernel(const float4* __restrict__ ro, const float4* __restrict__ rd,
                              const uint8_t* __restrict__ valid, int64_t n,
                              const int* __restrict__ bounds, uint32_t* __restrict__ keys,
                              int32_t* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vals[i] = (int32_t)i;
    keys[i] = valid && !valid[i] ? 0xffffffffu : morton_key(ro[i], rd[i], origin_box(bounds));
}

// Origin order: the origin's position along a 3-D Hilbert curve, 8 bits
// per axis over the batch's origin box in cubic cells (the box's largest
// extent on every axis, so that a flat spread of origins is not cut finer
// across its thin axis).  For shadow batches, whose directions all point at
// a light, this keeps a leaf's 32 origins close in space (image tiles put
// silhouette pixels' far-apart hit points together); unlike a Morton code,
// consecutive cells of the curve are always neighbours, so no leaf spans a
// jump.
__device__ __forceinline__ uint32_t origin_key(float4 o, const OriginBox& box) {
    uint32_t q[3];
    const float ov[3] = {o.x, o.y, o.z};
    float cube = 0.f;  // cubic cells: the largest extent on every axis
#pragma unroll
    for (int a = 0; a < 3; ++a) cube = fmaxf(cube, box.hi[a] - box.lo[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float ext = cube;
        constexpr float kCells = (float)(1 << kOriginAxisBits);
        float v = ext > 0.f ? (ov[a] - box.lo[a]) / ext * kCells : 0.f;
        v = fminf(fmaxf(v, 0.f), kCells - 1.f);  // NaN -> 0
        q[a] = (uint32_t)v;
    }
    hilbert3(q, kOriginAxisBits);
    return min(kMaxOriginKey, (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]));
}

__global__ void origin_key_kernel(const float4* __restrict__ ro, const uint8_t* __restrict__ valid,
                                  int64_t n, const int* __restrict__ bounds, uint32_t* __restrict__ keys,
                                  int32_t* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vals[i] = (int32_t)i;
    keys[i] = valid && !valid[i] ? 0xffffffffu : origin_key(ro[i], origin_box(bounds));
}

// Ray-image order: when the caller declared its batches as a W x H ray image
// (Preprocess, accelerators/rayhierarchy.cpp:250-265; ray i at x = i mod W,
// y = i div W), the key is the 2-D Morton code of (x, y), so a leaf of 32
// rays is an 8 x 4 tile of the image -- the reference's chunkX x chunkY
// leaves, but compact at every level above too.
__device__ __forceinline__ uint32_t spread16(uint32_t v) {
    v &= 0xffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

__device__ __forceinline__ uint32_t image_key(int64_t i, int64_t width) {
    const uint32_t x = (uint32_t)(i % width), y = (uint32_t)(i / width);
    // 15 bits per axis keeps valid keys below 0xffffffff
    return min(kMaxValidKey, (spread16(y & 0x7fffu) << 1) | spread16(x & 0x7fffu));
}

__global__ void image_key_kernel(const uint8_t* __restrict__ valid, int64_t n, int64_t width,
                                 uint32_t* __restrict__ keys, int32_t* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vals[i] = (int32_t)i;
    keys[i] = valid && !valid[i] ? 0xffffffffu : image_key(i, width);
}

// The same order without a sort, for a fully valid ray image whose width
// 2^a and height 2^b are powers of two: the Morton code of (x, y) then ranks
// every pixel densely -- the low min(a, b) bits of x and y interleaved, the
// longer side's remaining bits on top -- so ray i goes straight to its rank.
__global__ void image_perm_kernel(int64_t n, int a, int b, int32_t* __restrict__ perm_out,
                                  uint32_t* __restrict__ keys_out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t x = (uint32_t)(i & ((1ll << a) - 1)), y = (uint32_t)(i >> a);
    const int c = min(a, b);
    const uint32_t m = (1u << c) - 1u;
    const uint32_t low = spread16(x & m) | (spread16(y & m) << 1);
    const uint32_t high = a > b ? (x >> c) : (y >> c);
    const uint32_t rank = (high << (2 * c)) | low;
    perm_out[rank] = (int32_t)i;
    keys_out[rank] = min(kMaxValidKey, (spread16(y) << 1) | spread16(x));
}

// Pass 1: digit histogram of each tile, stored digit-major: hist[d * tiles + tile].
__global__ void __launch_bounds__(kSortThreads)
    radix_hist_kernel(const uint32_t* __restrict__ keys, int64_t n, int shift, int tiles,
                      uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kRadix];
    for (int k = threadIdx.x; k < kRadix; k += kSortThreads) h[k] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + (int64_t)k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & kDigitMask], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kRadix; k += kSortThreads)
        hist[(int64_t)k * tiles + blockIdx.x] = h[k];
}

// Pass 2: exclusive scan of the m = tiles*256 counts in three phases:
// per-chunk sums, one CTA over the chunk sums, per-chunk scans with offsets.
constexpr int kScanChunk = 4096;  // counts per chunk, 4 per thread

__device__ __forceinline__ uint32_t block_excl_scan_1024(uint32_t v, uint32_t* warp_sums,
                                                         uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warp_sums[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = (warp ? warp_sums[warp - 1] : 0u) + x - v;
    if (total) *total = warp_sums[31];
    return excl;
}

__global__ void __launch_bounds__(1024) scan_chunk_sums(const uint32_t* __restrict__ a, int64_t m,
                                                        uint32_t* __restrict__ sums) {
    __shared__ uint32_t ws[32];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk + threadIdx.x * 4;
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (base + k < m) v += a[base + k];
    uint32_t total;
    block_excl_scan_1024(v, ws, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) scan_top(uint32_t* __restrict__ sums, int nchunks) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nchunks; base += 1024) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < nchunks ? sums[i] : 0u;
        uint32_t total;
        const uint32_t e = block_excl_scan_1024(v, ws, &total);
        if (i < nchunks) sums[i] = carry + e;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(1024) scan_chunks(uint32_t* __restrict__ a, int64_t m,
                                                    const uint32_t* __restrict__ sums) {
    __shared__ uint32_t ws[32];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk + threadIdx.x * 4;
    uint32_t v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = base + k < m ? a[base + k] : 0u;
        s += v[k];
    }
    uint32_t run = sums[blockIdx.x] + block_excl_scan_1024(s, ws, nullptr);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < m) a[base + k] = run;
        run += v[k];
    }
}

// Up to kScanOne counts (16-byte aligned) in one CTA: one launch instead of
// three.
constexpr int kScanOne = 16384;

__global__ void __launch_bounds__(1024) scan_one(uint32_t* __restrict__ a, int m) {
    __shared__ uint32_t ws[32];
    constexpr int kQuads = kScanOne / 1024 / 4;
    uint4* a4 = reinterpret_cast<uint4*>(a);
    uint32_t v[4 * kQuads], s = 0;
#pragma unroll
    for (int k = 0; k < kQuads; ++k) {
        const int q = threadIdx.x * kQuads + k;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (4 * q + 3 < m) {
            x = a4[q];
        } else if (4 * q < m) {
            x.x = a[4 * q];
            x.y = 4 * q + 1 < m ? a[4 * q + 1] : 0u;
            x.z = 4 * q + 2 < m ? a[4 * q + 2] : 0u;
        }
        v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
        s += x.x + x.y + x.z + x.w;
    }
    uint32_t run = block_excl_scan_1024(s, ws, nullptr);
#pragma unroll
    for (int k = 0; k < kQuads; ++k) {
        const int q = threadIdx.x * kQuads + k;
        uint4 x;
        x.x = run; x.y = x.x + v[4 * k]; x.z = x.y + v[4 * k + 1]; x.w = x.z + v[4 * k + 2];
        run = x.w + v[4 * k + 3];
        if (4 * q + 3 < m) {
            a4[q] = x;
        } else if (4 * q < m) {
            a[4 * q] = x.x;
            if (4 * q + 1 < m) a[4 * q + 1] = x.y;
            if (4 * q + 2 < m) a[4 * q + 2] = x.z;
        }
    }
}

// Pass 3: stable scatter.  Element order inside a tile is (warp, item, lane),
// which is the original order, so ranks computed in that order keep the sort
// stable.
__global__ void __launch_bounds__(kSortThreads)
    radix_scatter_kernel(const uint32_t* __restrict__ keys, const int32_t* __restrict__ vals,
                         int64_t n, int shift, int tiles, const uint32_t* __restrict__ offs,
                         uint32_t* __restrict__ keys_out, int32_t* __restrict__ vals_out) {
    __shared__ uint32_t wcount[kSortWarps][kRadix];  // per-warp digit counts, then prefixes
    __shared__ uint32_t toff[kRadix];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kSortWarps * kRadix; k += kSortThreads)
        (&wcount[0][0])[k] = 0;
    for (int k = threadIdx.x; k < kRadix; k += kSortThreads)
        toff[k] = offs[(int64_t)k * tiles + blockIdx.x];
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile + (int64_t)warp * 32 * kSortItems;
    uint32_t key[kSortItems];
    int32_t val[kSortItems];
    uint32_t rank[kSortItems];
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + (int64_t)k * 32 + lane;
        const bool ok = i < n;
        key[k] = ok ? keys[i] : 0xffffffffu;
        val[k] = ok ? vals[i] : 0;
        const uint32_t dg = (key[k] >> shift) & kDigitMask;
        const uint32_t inb = __ballot_sync(0xffffffffu, ok);
        uint32_t peers = __match_any_sync(0xffffffffu, ok ? dg : (uint32_t)kRadix) & inb;
        if (!ok) peers = 0;
        const uint32_t before = wcount[warp][dg];
        __syncwarp();
        rank[k] = before + __popc(peers & lt);
        const int leader = peers ? __ffs(peers) - 1 : -1;
        if (ok && lane == leader) wcount[warp][dg] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Exclusive prefix over warps for every digit.
    for (int dg = threadIdx.x; dg < kRadix; dg += kSortThreads) {
        uint32_t run = 0;
        for (int w = 0; w < kSortWarps; ++w) {
            uint32_t c = wcount[w][dg];
            wcount[w][dg] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + (int64_t)k * 32 + lane;
        if (i >= n) continue;
        const uint32_t dg = (key[k] >> shift) & kDigitMask;
        const uint32_t pos = toff[dg] + wcount[warp][dg] + rank[k];
        keys_out[pos] = key[k];
        vals_out[pos] = val[k];
    }
}

// ------------------------------------------------- small batches: one cluster

// Up to kClusterKeys keys are sorted by one cluster of 8 or 16 CTAs in one
// launch: the keys and values stay in the CTAs' shared memory between
// passes, a pass exchanges the CTAs' digit counts and scatters through
// distributed shared memory, and the rays' keys (with the origin bounds) are
// computed on the way in.  The order is that of the passes above: a stable
// sort has only one.
//
// Bound by latency (barriers and shared memory round trips), so the passes
// are few: digits of 8 to 10 bits, and no bit above an image's keys.  A
// batch of 19,159 rays: about 26 us an order under the profiler, where the
// passes above took 90 (20 launches).
constexpr int kClusterCtas = 16;
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterItems = 8;  // keys per thread at most
constexpr int kClusterPer = kClusterThreads * kClusterItems;
constexpr int64_t kClusterKeys = (int64_t)kClusterCtas * kClusterPer;
constexpr int64_t kClusterSmall = 8192;
constexpr int kClusterDigit = 10;  // bits per digit at most (8 at least)
constexpr int kClusterRadix = 1 << kClusterDigit;

enum : int { kKeysGiven = 0, kKeysImage = 1, kKeysOrigin = 2, kKeysMorton = 3 };

struct SortSource {
    int mode = kKeysGiven;
    const uint32_t* keys = nullptr;  // kKeysGiven
    const int32_t* vals = nullptr;
    const float4 *o = nullptr, *d = nullptr;  // the rays otherwise
    const uint8_t* valid = nullptr;
    int64_t width = 0;          // kKeysImage
    uint4* cache = nullptr;     // kKeysOrigin: the kept (origin, mint) and validity
    uint8_t* vcache = nullptr;
};

struct ClusterSmem {
    uint2 kv[kClusterPer];  // (key, value)
    uint16_t wcount[kClusterWarps * kClusterRadix];  // [warp][digit]: counts, then prefixes
    uint32_t part[kClusterRadix], part2[kClusterRadix];  // [share][digit] sums
    uint32_t total[kClusterRadix];                   // this CTA's digit counts (read by the others)
    uint32_t toff[kClusterRadix];
    uint32_t ws[32];
    int bounds[8];                           // (read by the others)
};

__device__ __forceinline__ void cluster_arrive_wait() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(cta));
    return r;
}
__device__ __forceinline__ uint32_t cluster_load(const void* p, uint32_t cta) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_map(p, cta)) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_store(const void* p, uint32_t cta, uint2 v) {
    asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(cluster_map(p, cta)), "r"(v.x), "r"(v.y) : "memory");
}

// The lanes of the warp whose digit equals this lane's, among those with ok
// set (0 for the others): one vote per bit.  One warp's __match_any_sync takes
// some 55 cycles of its SM for distinct digits, the votes a third of that; the
// large batches' scatter, which waits for memory, is no faster for it (27 us a
// pass of 4 M keys, 30 with votes).
template <int MAXBITS>
__device__ __forceinline__ uint32_t digit_peers(uint32_t dg, bool ok, int bits) {
    uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int b = 0; b < MAXBITS; ++b) {
        if (b >= bits) break;
        const uint32_t v = __ballot_sync(0xffffffffu, (dg >> b) & 1u);
        peers &= (dg >> b) & 1u ? v : ~v;
    }
    return ok ? peers : 0u;
}

// CTA c holds positions [c * per, c * per + per) of the n keys, its warp w
// the next 32 * items of them; per is at most 1024 * items.
__global__ void __launch_bounds__(kClusterThreads, 1)
    sort_cluster_kernel(SortSource src, int n, int per, int items, int bits, int digit_bits,
                        uint32_t* __restrict__ keys_out, int32_t* __restrict__ vals_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem& sm = *reinterpret_cast<ClusterSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t cta = blockIdx.x;  // one cluster: the rank in it
    const int base = (int)cta * per;
    const int cnt = max(0, min(per, n - base));
    const unsigned full = 0xffffffffu;

    OriginBox box{};
    if (src.mode >= kKeysOrigin) {
        if (tid < 6) sm.bounds[tid] = tid < 3 ? 0x7fffffff : (int)0x80000000;
        __syncthreads();
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int j = tid; j < cnt; j += kClusterThreads) {
            const uint8_t v = src.valid ? (src.valid[base + j] != 0) : 1;
            uint4 e = make_uint4(0u, 0u, 0u, 0u);
            if (v) {
                const float4 o = src.o[base + j];
                e = make_uint4(__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), __float_as_uint(o.w));
                if (isfinite(o.x) && isfinite(o.y) && isfinite(o.z)) {
                    lo[0] = fminf(lo[0], o.x); lo[1] = fminf(lo[1], o.y); lo[2] = fminf(lo[2], o.z);
                    hi[0] = fmaxf(hi[0], o.x); hi[1] = fmaxf(hi[1], o.y); hi[2] = fmaxf(hi[2], o.z);
                }
            }
            if (src.cache) {
                src.cache[base + j] = e;
                src.vcache[base + j] = v;
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int l = __reduce_min_sync(full, ord_f(lo[a])), h = __reduce_max_sync(full, ord_f(hi[a]));
            if (lane == 0) {
                atomicMin(&sm.bounds[a], l);
                atomicMax(&sm.bounds[3 + a], h);
            }
        }
        __syncthreads();
        cluster_arrive_wait();
        int b[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            b[a] = (int)cluster_load(&sm.bounds[a], (uint32_t)lane & (gridDim.x - 1u));
            b[a] = a < 3 ? __reduce_min_sync(full, b[a]) : __reduce_max_sync(full, b[a]);
        }
        box = origin_box(b);
    }
    for (int j = tid; j < cnt; j += kClusterThreads) {
        const int i = base + j;
        uint32_t key = 0xffffffffu;
        if (src.mode == kKeysGiven)
            key = src.keys[i];
        else if (!(src.valid && !src.valid[i]))
            key = src.mode == kKeysImage    ? image_key(i, src.width)
                  : src.mode == kKeysOrigin ? origin_key(src.o[i], box)
                                            : morton_key(src.o[i], src.d[i], box);
        sm.kv[j] = make_uint2(key, (uint32_t)(src.mode == kKeysGiven ? src.vals[i] : i));
    }

    const uint32_t lt = (1u << lane) - 1u;
    // a digit's sums are shared out to 1024 >> digit_bits threads
    const int radix = 1 << digit_bits;
    const int dgt = tid & (radix - 1), share = tid >> digit_bits, shares = kClusterThreads >> digit_bits;
    const int warps = kClusterWarps / shares, ctas = (int)gridDim.x / shares;
    uint16_t* mycount = sm.wcount + warp * radix;
    for (int shift = 0; shift < bits; shift += digit_bits) {
        const bool last = shift + digit_bits >= bits;
        for (int k = tid; k < kClusterWarps * radix / 2; k += kClusterThreads)
            reinterpret_cast<uint32_t*>(sm.wcount)[k] = 0;
        __syncthreads();
        uint32_t key[kClusterItems], rank[kClusterItems];
        int32_t val[kClusterItems];
#pragma unroll
        for (int k = 0; k < kClusterItems; ++k) {
            if (k >= items) break;
            const int j = (warp * items + k) * 32 + lane;
            const bool ok = j < cnt;
            const uint2 e = ok ? sm.kv[j] : make_uint2(0xffffffffu, 0u);
            key[k] = e.x;
            val[k] = (int32_t)e.y;
            const uint32_t dg = (key[k] >> shift) & (radix - 1);
            if ((warp * items + k) * 32 >= cnt) continue;  // whole warp
            const uint32_t peers = digit_peers<kClusterDigit>(dg, ok, digit_bits);
            const uint32_t before = mycount[dg];
            __syncwarp();
            rank[k] = before + __popc(peers & lt);
            if (ok && (peers & lt) == 0) mycount[dg] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // exclusive prefix over the warps for every digit
        uint16_t* col = sm.wcount + share * warps * radix + dgt;
        uint32_t run = 0;
        if (shares > 1) {
            uint32_t sum = 0;
#pragma unroll 8
            for (int w = 0; w < warps; ++w) sum += col[w * radix];
            sm.part[tid] = sum;
            __syncthreads();
            for (int p = 0; p < share; ++p) run += sm.part[p * radix + dgt];
        }
#pragma unroll 8
        for (int w = 0; w < warps; ++w) {
            const uint32_t c = col[w * radix];
            col[w * radix] = (uint16_t)run;
            run += c;
        }
        if (share == shares - 1) sm.total[dgt] = run;
        cluster_arrive_wait();  // every CTA's counts; every key is in registers
        // keys of this digit in the CTAs before this one, and in all
        uint32_t mine = 0, all = 0;
#pragma unroll 8
        for (int k = 0; k < ctas; ++k) {
            const uint32_t c = (uint32_t)(share * ctas + k), v = cluster_load(&sm.total[dgt], c);
            all += v;
            mine += c < cta ? v : 0u;
        }
        if (shares > 1) {
            sm.part[tid] = mine;
            sm.part2[tid] = all;
            __syncthreads();
            if (share == 0)
                for (int p = 1; p < shares; ++p) {
                    mine += sm.part[p * radix + dgt];
                    all += sm.part2[p * radix + dgt];
                }
        }
        const uint32_t before_digit = block_excl_scan_1024(share == 0 ? all : 0u, sm.ws, nullptr);
        if (share == 0) sm.toff[dgt] = before_digit + mine;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kClusterItems; ++k) {
            if (k >= items) break;
            const int j = (warp * items + k) * 32 + lane;
            if (j >= cnt) continue;
            const uint32_t dg = (key[k] >> shift) & (radix - 1);
            const uint32_t pos = sm.toff[dg] + mycount[dg] + rank[k];
            if (last) {
                keys_out[pos] = key[k];
                vals_out[pos] = val[k];
            } else {
                const uint32_t to = pos / (uint32_t)per, at = pos - to * (uint32_t)per;
                cluster_store(&sm.kv[at], to, make_uint2(key[k], (uint32_t)val[k]));
            }
        }
        cluster_arrive_wait();  // keys have arrived; no CTA leaves while its counts are read
    }
}

// Per-device settings (cheap, idempotent): set on every call so that each
// device the library launches on has them.
static cudaError_t sort_cluster_attributes() {
    const cudaError_t e = cudaFuncSetAttribute(sort_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(ClusterSmem));
    return e != cudaSuccess ? e : cudaFuncSetAttribute(sort_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

// Keys that one cluster of the device can sort: half where it has no room for
// 16 CTAs (more than the portable size, so not promised).
static int64_t cluster_keys(int device) {
    static std::atomic<int> fits[64];  // 0 not asked yet, 1 no, 2 yes
    if (device < 0 || device >= 64) return kClusterKeys / 2;
    if (fits[device].load() == 0) {
        cudaLaunchAttribute dims{};
        dims.id = cudaLaunchAttributeClusterDimension;
        dims.val.clusterDim.x = kClusterCtas;
        dims.val.clusterDim.y = dims.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kClusterCtas);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = sizeof(ClusterSmem);
        cfg.attrs = &dims;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool ok = sort_cluster_attributes() == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, sort_cluster_kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        fits[device].store(ok ? 2 : 1);
    }
    return fits[device].load() == 2 ? kClusterKeys : kClusterKeys / 2;
}

// One cluster sorts the n <= cluster_keys() keys of src into (keys_out, vals_out).
static int sort_cluster(pbg_scene* s, const SortSource& src, int64_t n, int bits, uint32_t* keys_out, int32_t* vals_out,
                        cudaStream_t st) {
    PBG_CUDA(sort_cluster_attributes());
    // The most keys take the widest cluster; up to kClusterSmall, where an
    // 8-CTA cluster's barriers are the shorter part, half of it (frames of
    // 1,200 / 19,159 / 65,280 rays: 163 / 229 / 380 us with 8 CTAs, 172 / 228 /
    // 356 with 16).
    const int ctas = n <= kClusterSmall || cluster_keys(s->device) < kClusterKeys ? kClusterCtas / 2 : kClusterCtas;
    const int per = (int)(((n + ctas - 1) / ctas + 31) / 32 * 32);
    const int items = (per + kClusterThreads - 1) / kClusterThreads;
    if (src.mode == kKeysImage) {  // the keys' own bits, and one above them where invalid rays sort last
        int64_t side = src.width, rows = (n + src.width - 1) / src.width;
        int used = src.valid ? 1 : 0;
        for (int64_t m = std::max(side, rows); m > 1; m = (m + 1) / 2) used += 2;
        bits = std::min(bits, std::max(used, 1));
    }
    const int passes = (bits + kClusterDigit - 1) / kClusterDigit;
    const int digit_bits = std::max(8, (bits + passes - 1) / passes);
    prof_begin(s, st);
    cudaLaunchAttribute dims{};
    dims.id = cudaLaunchAttributeClusterDimension;
    dims.val.clusterDim.x = (unsigned)ctas;
    dims.val.clusterDim.y = dims.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem);
    cfg.stream = st;
    cfg.attrs = &dims;
    cfg.numAttrs = 1;
    PBG_CUDA(cudaLaunchKernelEx(&cfg, sort_cluster_kernel, src, (int)n, per, items, bits, digit_bits, keys_out, vals_out));
    prof_end(s, st, kStageSort, 1);
    return PBG_OK;
}

// Words of radix_sort_pairs' histogram buffer for n keys: the counts, eight
// words for bounds, the scan's chunk sums.
size_t radix_hist_words(int64_t n) {
    const size_t m = (size_t)((n + kSortTile - 1) / kSortTile) * kRadix;
    return m + 8 + (m + kScanChunk - 1) / kScanChunk + 8;
}

// Sorts (keys, vals) of length n in place through the tmp buffers; returns
// pointers to the sorted arrays (which alternate between the two buffers).
int radix_sort_pairs(pbg_scene* s, uint32_t* keys, int32_t* vals, uint32_t* keys_tmp, int32_t* vals_tmp,
                     uint32_t* hist, int64_t n, int bits, uint32_t** keys_out, int32_t** vals_out,
                     cudaStream_t st) {
    if (n > 0 && n <= cluster_keys(s->device)) {
        SortSource src;
        src.keys = keys;
        src.vals = vals;
        *keys_out = keys_tmp;
        *vals_out = vals_tmp;
        return sort_cluster(s, src, n, bits, keys_tmp, vals_tmp, st);
    }
    const int tiles = (int)((n + kSortTile - 1) / kSortTile);
    uint32_t *ka = keys, *kb = keys_tmp;
    int32_t *va = vals, *vb = vals_tmp;
    for (int shift = 0; shift < bits; shift += kDigitBits) {
        prof_begin(s, st);
        radix_hist_kernel<<<tiles, kSortThreads, 0, st>>>(ka, n, shift, tiles, hist);
        prof_end(s, st, kStageSort, 1);
        const int64_t m = (int64_t)tiles * kRadix;
        const int nchunks = (int)((m + kScanChunk - 1) / kScanChunk);
        uint32_t* sums = hist + m + 8;  // after the histogram and the bounds words
        prof_begin(s, st);
        scan_chunk_sums<<<nchunks, 1024, 0, st>>>(hist, m, sums);
        scan_top<<<1, 1024, 0, st>>>(sums, nchunks);
        scan_chunks<<<nchunks, 1024, 0, st>>>(hist, m, sums);
        prof_end(s, st, kStageSort, 3);
        prof_begin(s, st);
        radix_scatter_kernel<<<tiles, kSortThreads, 0, st>>>(ka, va, n, shift, tiles, hist, kb, vb);
        prof_end(s, st, kStageSort, 1);
        PBG_CUDA(cudaGetLastError());
        uint32_t* tk = ka; ka = kb; kb = tk;
        int32_t* tv = va; va = vb; vb = tv;
    }
    *keys_out = ka;
    *vals_out = va;
    return PBG_OK;
}

// Computes the order of a batch (image, Hilbert origin or 6-D Morton).  *perm (device, n entries) lists ray
// indices in sorted order; valid rays come first.
// Shadow batches of one frame (one per light sample) leave from the same
// points (the same origin and mint) with the same validity, so their origin
// order repeats.  compare_origins_kernel sets *moved at any ray whose
// validity, or whose (origin, mint) while valid, differs bit for bit from
// the cached batch, and stores the new entry in the cache;
// store_sorted_kernel keeps a fresh sort's order for the next batch.
__global__ void compare_origins_kernel(const float4* __restrict__ ro, const uint8_t* __restrict__ valid,
                                       int64_t n, uint4* __restrict__ cache, uint8_t* __restrict__ vcache,
                                       int* __restrict__ moved) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t v = valid ? (valid[i] != 0) : 1;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if (v) {
        const float4 o = ro[i];
        e = make_uint4(__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), __float_as_uint(o.w));
    }
    const uint4 c = cache[i];
    if (vcache[i] != v || c.x != e.x || c.y != e.y || c.z != e.z || c.w != e.w) {
        *moved = 1;
        cache[i] = e;
        vcache[i] = v;
    }
}

__global__ void store_sorted_kernel(const uint32_t* __restrict__ skeys, const int32_t* __restrict__ perm,
                                    int64_t n, uint32_t* __restrict__ skeys_cache,
                                    int32_t* __restrict__ perm_cache) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    skeys_cache[i] = skeys[i];
    perm_cache[i] = perm[i];
}

static bool pow2_le(int64_t v, int64_t cap) { return v > 0 && v <= cap && (v & (v - 1)) == 0; }

int ray_sort(pbg_scene* s, const float4* o, const float4* d, const uint8_t* valid, int64_t n,
             const int32_t** perm, const uint32_t** sorted_keys, cudaStream_t st, int order) {
    Work& w = s->work;
    const int tiles = (int)((n + kSortTile - 1) / kSortTile);
    int rc;
    if ((rc = ensure(w.mkeys, (size_t)n * 4)) || (rc = ensure(w.mkeys_tmp, (size_t)n * 4)) ||
        (rc = ensure(w.perm, (size_t)n * 4)) || (rc = ensure(w.perm_tmp, (size_t)n * 4)) ||
        (rc = ensure(w.hist, radix_hist_words(n) * 4)))
        return rc;
    int* bounds = (int*)((uint32_t*)w.hist.ptr + (size_t)tiles * kRadix);
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    int64_t blocks = (n + 255) / 256;
    if (blocks > 4 * sms) blocks = 4 * sms;
    w.origin_reused = false;
    w.origin_speculative = false;
    if (order == kOrderOrigin) {
        // reuse the previous origin order when origins and validity repeat
        const void* before[4] = {w.origin_cache.ptr, w.osort_keys.ptr, w.osort_perm.ptr,
                                 w.origin_valid.ptr};
        const bool was_cached = w.origin_sort_n == n;
        w.origin_sort_n = -1;  // set again only once the cache is consistent
        if ((rc = ensure(w.origin_cache, (size_t)n * 16)) || (rc = ensure(w.osort_keys, (size_t)n * 4)) ||
            (rc = ensure(w.osort_perm, (size_t)n * 4)) || (rc = ensure(w.origin_valid, (size_t)n)))
            return rc;
        const bool comparable = was_cached && before[0] == w.origin_cache.ptr &&
                                before[1] == w.osort_keys.ptr && before[2] == w.osort_perm.ptr &&
                                before[3] == w.origin_valid.ptr;
        if (!comparable && n <= cluster_keys(s->device)) {
            SortSource src;
            src.mode = kKeysOrigin;
            src.o = o;
            src.valid = valid;
            src.cache = (uint4*)w.origin_cache.ptr;
            src.vcache = (uint8_t*)w.origin_valid.ptr;
            rc = sort_cluster(s, src, n, kOriginKeyBits, (uint32_t*)w.osort_keys.ptr, (int32_t*)w.osort_perm.ptr, st);
            if (rc) return rc;
            w.origin_sort_n = n;
            *perm = (const int32_t*)w.osort_perm.ptr;
            if (sorted_keys) *sorted_keys = (const uint32_t*)w.osort_keys.ptr;
            return PBG_OK;
        }
        int* moved = (int*)s->err.ptr + kStatusOriginMoved;
        PBG_CUDA(cudaMemsetAsync(moved, 0, sizeof(int), st));
        prof_begin(s, st);
        compare_origins_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            o, valid, n, (uint4*)w.origin_cache.ptr, (uint8_t*)w.origin_valid.ptr, moved);
        prof_end(s, st, kStageSort, 1);
        PBG_CUDA(cudaGetLastError());
        if (comparable) {
            // The kept order is taken without waiting for the comparison:
            // the batch's closing status read carries *moved, and a batch
            // whose origins moved is traced again with a fresh sort.
            w.origin_sort_n = n;
            w.origin_reused = true;
            w.origin_speculative = true;
            *perm = (const int32_t*)w.osort_perm.ptr;
            if (sorted_keys) *sorted_keys = (const uint32_t*)w.osort_keys.ptr;
            return PBG_OK;
        }
        prof_begin(s, st);
        init_bounds_kernel<<<1, 32, 0, st>>>(bounds);
        origin_bounds_kernel<<<(unsigned)blocks, 256, 0, st>>>(o, valid, n, bounds);
        prof_end(s, st, kStageSort, 2);
        prof_begin(s, st);
        origin_key_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            o, valid, n, bounds, (uint32_t*)w.mkeys.ptr, (int32_t*)w.perm.ptr);
        prof_end(s, st, kStageSort, 1);
    } else if (s->image_w > 0 && n == s->image_w * s->image_h && valid == nullptr &&
               pow2_le(s->image_w, 1 << 15) && pow2_le(s->image_h, 1 << 15)) {
        int a = 0, b = 0;
        while ((1ll << a) < s->image_w) ++a;
        while ((1ll << b) < s->image_h) ++b;
        prof_begin(s, st);
        image_perm_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            n, a, b, (int32_t*)w.perm_tmp.ptr, (uint32_t*)w.mkeys_tmp.ptr);
        prof_end(s, st, kStageSort, 1);
        PBG_CUDA(cudaGetLastError());
        *perm = (const int32_t*)w.perm_tmp.ptr;
        if (sorted_keys) *sorted_keys = (const uint32_t*)w.mkeys_tmp.ptr;
        return PBG_OK;
    } else if (n <= cluster_keys(s->device)) {
        SortSource src;
        src.mode = s->image_w > 0 && n == s->image_w * s->image_h ? kKeysImage : kKeysMorton;
        src.o = o;
        src.d = d;
        src.valid = valid;
        src.width = s->image_w;
        *perm = (const int32_t*)w.perm_tmp.ptr;
        if (sorted_keys) *sorted_keys = (const uint32_t*)w.mkeys_tmp.ptr;
        return sort_cluster(s, src, n, kKeyBits, (uint32_t*)w.mkeys_tmp.ptr, (int32_t*)w.perm_tmp.ptr, st);
    } else if (s->image_w > 0 && n == s->image_w * s->image_h) {
        prof_begin(s, st);
        image_key_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            valid, n, s->image_w, (uint32_t*)w.mkeys.ptr, (int32_t*)w.perm.ptr);
        prof_end(s, st, kStageSort, 1);
    } else {
        prof_begin(s, st);
        init_bounds_kernel<<<1, 32, 0, st>>>(bounds);
        origin_bounds_kernel<<<(unsigned)blocks, 256, 0, st>>>(o, valid, n, bounds);
        prof_end(s, st, kStageSort, 2);
        prof_begin(s, st);
        morton_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
            o, d, valid, n, bounds, (uint32_t*)w.mkeys.ptr, (int32_t*)w.perm.ptr);
        prof_end(s, st, kStageSort, 1);
    }
    PBG_CUDA(cudaGetLastError());
    uint32_t* ko;
    int32_t* vo;
    // The bounds words sit after the histogram; 8-bit passes over the low
    // 24 (origin) or 30 key bits, invalid rays last (kMaxValidKey).  An
    // origin order alternates with the kept-order buffers, so that its odd
    // number of passes ends in them.
    const bool origin = order == kOrderOrigin;
    rc = radix_sort_pairs(s, (uint32_t*)w.mkeys.ptr, (int32_t*)w.perm.ptr,
                          (uint32_t*)(origin ? w.osort_keys.ptr : w.mkeys_tmp.ptr),
                          (int32_t*)(origin ? w.osort_perm.ptr : w.perm_tmp.ptr), (uint32_t*)w.hist.ptr, n,
                          origin ? kOriginKeyBits : kKeyBits, &ko, &vo, st);
    if (rc) return rc;
    if (origin) {
        if (ko != (uint32_t*)w.osort_keys.ptr) {  // an even number of passes
            prof_begin(s, st);
            store_sorted_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
                ko, vo, n, (uint32_t*)w.osort_keys.ptr, (int32_t*)w.osort_perm.ptr);
            prof_end(s, st, kStageSort, 1);
            PBG_CUDA(cudaGetLastError());
            ko = (uint32_t*)w.osort_keys.ptr;
            vo = (int32_t*)w.osort_perm.ptr;
        }
        w.origin_sort_n = n;
    }
    *perm = vo;
    if (sorted_keys) *sorted_keys = ko;
    return PBG_OK;
}

// In-place exclusive scan of m counts (the renderer's queue compaction).
int scan_counts(pbg_scene* s, uint32_t* a, int64_t m, cudaStream_t st) {
    if (m <= 0) return PBG_OK;
    if (m <= kScanOne && ((uintptr_t)a & 15u) == 0) {
        scan_one<<<1, 1024, 0, st>>>(a, (int)m);
        s->counters.kernel_launches++;
        PBG_CUDA(cudaGetLastError());
        return PBG_OK;
    }
    const int nchunks = (int)((m + kScanChunk - 1) / kScanChunk);
    int rc = ensure(s->work.scan_sums, (size_t)(nchunks + 8) * 4);
    if (rc) return rc;
    uint32_t* sums = (uint32_t*)s->work.scan_sums.ptr;
    scan_chunk_sums<<<nchunks, 1024, 0, st>>>(a, m, sums);
    scan_top<<<1, 1024, 0, st>>>(sums, nchunks);
    scan_chunks<<<nchunks, 1024, 0, st>>>(a, m, sums);
    s->counters.kernel_launches += 3;
    PBG_CUDA(cudaGetLastError());
    return PBG_OK;
}

int ray_order(pbg_scene* s, const float4* o, const float4* d, int64_t n, const int32_t** perm,
              cudaStream_t st) {
    if (n < 4096) {  // too small to gain from ordering
        *perm = nullptr;
        return PBG_OK;
    }
    return ray_sort(s, o, d, nullptr, n, perm, nullptr, st, kOrderDefault);
}

}  // namespace pbg
