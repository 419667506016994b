// pbg_train.cu -- one SGD step of the learned traversal ordering.
//
// train_kernel runs the whole forward and backward pass of a 128-record tile
// in one CTA: features and weights are staged in shared memory once, the
// three forward products, the two backward products and the three weight
// gradients are tcgen05 MMAs with FP32 accumulators in tensor memory, and
// nothing between them leaves the SM.  The gradients contract over the
// records, so their operands are the tiles already in shared memory read
// transposed (MN-major descriptors): no transposed copies are made.  A CTA
// that gets several tiles keeps accumulating its weight gradients in tensor
// memory; each CTA then writes one partial gradient, and apply_kernel sums
// the partials in CTA order (a fixed order: the same records give the same
// bits) and updates the parameters.
//
// What bounds it: eight MMA -> TMEM read -> shared memory round trips of
// about a microsecond each in one CTA per 128 records; the tensor pipe is
// nearly idle.  The step it replaces ran each product, transpose, bias,
// column sum and reduction as its own kernel (32 launches a step).  8 steps
// of 8,192 records through pbg_learn_train, weights read back: 2,700 us
// before, 228 us now (23 us a step on the device, 64 of 152 SMs).
//
// TMEM columns (512, one CTA per SM): [0, 256) the products in flight (layer
// 1 at 0, layer 2 at 64, logits at 0 once both are read, dH2 at 0, dH1 at
// 64); [256, 384) dW3 as two 128-cluster halves; [384, 448) [dZ2 | dZ1]^T H1,
// whose first 64 lanes are dW2; [448, 512) X^T dZ1, the transpose of dW1.
#include <algorithm>

#include "pbg_internal.h"
#include "pbg_learn.h"
#include "pbg_quotient.h"
#include "pbg_tc.cuh"

namespace pbg {

namespace {

constexpr int kTrainThreads = 512;  // four warps per quarter of the accumulator's lanes
constexpr int kTile = 128;          // records per tile
constexpr int kXCols = 128;         // feature columns staged (112 and zeros): M of X^T dZ1
constexpr int kDCols = 2 * kHidden; // [dZ2 | dZ1]

constexpr size_t kTX = (size_t)kTile * kXCols * 2, kTW1 = (size_t)kHidden * kFeat * 2, kTW2 = (size_t)kHidden * kHidden * 2,
                 kTW3 = (size_t)kClusters * kHidden * 2, kTH = (size_t)kTile * kHidden * 2, kTD = (size_t)kTile * kDCols * 2,
                 kTG = (size_t)kTile * kClusters * 2;
constexpr size_t kTrainSmem = kTX + kTW1 + kTW2 + kTW3 + 2 * kTH + kTD + kTG + (kHidden * 2 + kClusters) * 4 +
                              2 * 4 * kTile * 4 + 4 * kClusters * 4 + 64;
static_assert(kTrainSmem <= 227 * 1024, "one CTA's shared memory");

// Sums over the warp's 32 lanes of 16 values per lane by halving exchanges,
// 16 shuffles instead of 80: lanes 2 c and 2 c + 1 end with column c's sum.
__device__ __forceinline__ float column_sums(float* v, int lane) {
#pragma unroll
    for (int n = 8; n; n >>= 1) {
        const bool up = (lane & (2 * n)) != 0;
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const float send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__device__ __forceinline__ void put_group(uint8_t* dst, int r, int c, int cols, const float* v) {
    *(uint4*)(dst + core_offset(r, c, cols)) = pack8(v);
}

// The softmax's sixteen columns per step: eight from c, eight from c + 32.
__device__ __forceinline__ int column_of(int j) { return j < 8 ? j : 24 + j; }

// Those logits of this thread's record: the product in TMEM and the bias.
__device__ __forceinline__ void load_logits(float* v, uint32_t tl, const float* bias, int c) {
    tmem_ld8x2(tl + (uint32_t)c, tl + (uint32_t)c + 32u, v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 w = *(const float4*)(bias + c + column_of(4 * k));
        v[4 * k] += w.x;
        v[4 * k + 1] += w.y;
        v[4 * k + 2] += w.z;
        v[4 * k + 3] += w.w;
    }
}

// Row-major [ROWS x K] bf16 from global into a core-matrix tile COLS wide, by
// 16-byte asynchronous copies (all in flight at once; the caller waits).
template <int ROWS, int K, int COLS>
__device__ __forceinline__ void stage_tile(uint8_t* dst, const uint16_t* src) {
    for (int idx = threadIdx.x; idx < ROWS * (K / 8); idx += kTrainThreads) {
        const int r = idx / (K / 8), g = idx % (K / 8);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst + core_offset(r, g * 8, COLS))),
                     "l"(src + (size_t)r * K + g * 8)
                     : "memory");
    }
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Programmatic dependent launch: once the predecessor is complete and its
// writes are visible, this grid's successor may start (as soon as every CTA
// has come here).  In this order no more than one grid waits beside the one
// that works; released before its own wait, a grid of a later step could
// start, and its SM's L1 fill with an earlier step's lines, while the step
// between them was still to write them.
__device__ __forceinline__ void grid_dependency_wait_and_release() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// What a grid that this one overlaps has written: from L2, and not before the
// wait above (volatile, no const __restrict__ on the pointer, so neither the
// compiler nor an L1 line from before the wait can answer it).
__device__ __forceinline__ float load_written(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

// A tile [rows x cols] used with its columns along K (as stored) or with its
// rows along K (transposed: MN-major), from K step ks (16 elements of K each).
__device__ __forceinline__ uint64_t along_cols(const uint8_t* t, int cols, int ks) {
    return smem_desc(t + ks * 256, 128u, (uint32_t)(cols >> 3) * 128u);
}
__device__ __forceinline__ uint64_t along_rows(const uint8_t* t, int cols, int ks, int first_col = 0) {
    const uint32_t group = (uint32_t)(cols >> 3) * 128u;  // bytes from one eight-row group to the next
    return smem_desc(t + (size_t)ks * 2 * group + (first_col >> 3) * 128, group, 128u);
}
constexpr uint32_t kAT = 1u << 15, kBT = 1u << 16;  // instruction descriptor: A / B is MN-major

__global__ void __launch_bounds__(kTrainThreads, 1)
    train_kernel(const uint16_t* __restrict__ X, const int32_t* __restrict__ label, int tiles,
                 const uint16_t* Wb, const float* P, float scale, float* part, int* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sX = smem;
    uint8_t* sW1 = sX + kTX;
    uint8_t* sW2 = sW1 + kTW1;
    uint8_t* sW3 = sW2 + kTW2;
    uint8_t* sH1 = sW3 + kTW3;
    uint8_t* sH2 = sH1 + kTH;
    uint8_t* sD = sH2 + kTH;
    uint8_t* sG = sD + kTD;
    float* sb1 = (float*)(sG + kTG);
    float* sb2 = sb1 + kHidden;
    float* sb3 = sb2 + kHidden;
    float* smax = sb3 + kClusters;       // [4][128] a row's maximum in each column quarter
    int* sarg = (int*)(smax + 4 * kTile);
    float* scol = (float*)(sarg + 4 * kTile);  // [4][256] column sums of each lane quarter
    float* spart = (float*)sG;           // [32][128] partial sums of the softmax, before dZ3
    float* scol2 = smax;                 // [4][64], [4][64]: once the softmax is done
    float* scol1 = smax + 4 * kHidden;
    uint64_t* bar = (uint64_t*)(scol + 4 * kClusters);
    uint32_t* tslot = (uint32_t*)(bar + 1);
    float* sred = scol;                  // the CTA's loss and accuracy, at the end

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = warp & 3, g = warp >> 2;  // lane quarter, column group
    const int r = q * 32 + lane;            // this thread's record of the tile
    if (warp == 0) tmem_alloc(tslot, 512);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    // The launch overlaps the previous step's update (programmatic dependent
    // launch): what does not depend on it goes first -- the first tile's
    // features, barriers, tensor memory -- then the wait, then the weights.
    stage_tile<kTile, kFeat, kXCols>(sX, X + (size_t)blockIdx.x * kTile * kFeat);
    grid_dependency_wait_and_release();
    stage_tile<kHidden, kFeat, kFeat>(sW1, Wb + kOffW1);
    stage_tile<kHidden, kHidden, kHidden>(sW2, Wb + kOffW2);
    stage_tile<kClusters, kHidden, kHidden>(sW3, Wb + kOffW3);
    if (threadIdx.x < kTile * 2)  // the padding columns of X stay zero
        *(uint4*)(sX + core_offset(threadIdx.x >> 1, kFeat + 8 * (threadIdx.x & 1), kXCols)) = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < kHidden) {
        sb1[threadIdx.x] = load_written(P + kOffB1 + threadIdx.x);
        sb2[threadIdx.x] = load_written(P + kOffB2 + threadIdx.x);
    }
    if (threadIdx.x < kClusters) sb3[threadIdx.x] = load_written(P + kOffB3 + threadIdx.x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    const uint32_t tl = tbase + ((uint32_t)(q * 32) << 16);
    uint32_t phase = 0;
    // operands written by the generic proxy become visible to the MMAs, and
    // TMEM reads are ordered before the MMAs that overwrite them
    auto publish = [&]() {
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    };
    // all threads agree whether the wait was good
    auto await = [&]() -> bool {
        const bool ok = mbar_wait_bounded(bar, phase, status);
        phase ^= 1u;
        tc_fence_after();
        return __syncthreads_or(ok ? 0 : 1) == 0;
    };
    float loss = 0.f, right = 0.f, gb3 = 0.f, gb21 = 0.f;
    bool ok = true;
    uint32_t acc = 0;  // the weight gradients accumulate from the second tile on
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        if (tile != (int)blockIdx.x) stage_tile<kTile, kFeat, kXCols>(sX, X + (size_t)tile * kTile * kFeat);
        const int y = label[(size_t)tile * kTile + r];
        stage_wait();
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kFeat / 16; ++ks)
                tc_mma(tbase, along_cols(sX, kXCols, ks), along_cols(sW1, kFeat, ks), idesc_bf16(kTile, kHidden), ks > 0);
            tc_commit(bar);
        }
        if (!(ok = await())) break;
        float v[16];
        uint32_t live1 = 0, live2 = 0;  // which of this thread's hidden units are on
        tmem_ld16(tl + 16u * g, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            v[j] = fmaxf(v[j] + sb1[16 * g + j], 0.f);
            live1 |= v[j] > 0.f ? 1u << j : 0u;
        }
        put_group(sH1, r, 16 * g, kHidden, v);
        put_group(sH1, r, 16 * g + 8, kHidden, v + 8);
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kHidden / 16; ++ks)
                tc_mma(tbase + 64, along_cols(sH1, kHidden, ks), along_cols(sW2, kHidden, ks), idesc_bf16(kTile, kHidden), ks > 0);
            tc_commit(bar);
        }
        if (!(ok = await())) break;
        tmem_ld16(tl + 64u + 16u * g, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            v[j] = fmaxf(v[j] + sb2[16 * g + j], 0.f);
            live2 |= v[j] > 0.f ? 1u << j : 0u;
        }
        put_group(sH2, r, 16 * g, kHidden, v);
        put_group(sH2, r, 16 * g + 8, kHidden, v + 8);
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kHidden / 16; ++ks)
                tc_mma(tbase, along_cols(sH2, kHidden, ks), along_cols(sW3, kHidden, ks), idesc_bf16(kTile, kClusters), ks > 0);
            tc_commit(bar);
        }
        if (!(ok = await())) break;
        // Softmax over the record's 256 logits: this thread has columns 32 k +
        // 8 g .. + 7, two k at a time from TMEM in each of three passes
        // (unrolled over all 64 the code outgrows the instruction cache: 41 us
        // a launch, 5.6 of 18 cycles per instruction waiting for
        // instructions); the exponentials wait in TMEM between the second and
        // the third.
        float mx = -INFINITY;
        int am = 0;
#pragma unroll 1
        for (int c = 8 * g; c < kClusters; c += 64) {
            load_logits(v, tl, sb3, c);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (v[j] > mx) {
                    mx = v[j];
                    am = c + column_of(j);
                }
            }
        }
        smax[g * kTile + r] = mx;
        sarg[g * kTile + r] = am;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float om = smax[k * kTile + r];
            const int oa = sarg[k * kTile + r];
            if (om > mx || (om == mx && oa < am)) {
                mx = om;
                am = oa;
            }
        }
        // the sum: columns 32 apart first, then 16, 8, 4, 2 and 1 apart
        float lsum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int c = 8 * g; c < kClusters; c += 64) {
            load_logits(v, tl, sb3, c);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                v[j] = __expf(v[j] - mx);
                lsum[j & 7] += v[j];
            }
            tmem_st8x2(tl + (uint32_t)c, tl + (uint32_t)c + 32u, v);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) spart[(g * 8 + j) * kTile + r] = lsum[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 8; ++j)
            lsum[j] = (spart[j * kTile + r] + spart[(16 + j) * kTile + r]) +
                      (spart[(8 + j) * kTile + r] + spart[(24 + j) * kTile + r]);
        const float s = ((lsum[0] + lsum[4]) + (lsum[2] + lsum[6])) + ((lsum[1] + lsum[5]) + (lsum[3] + lsum[7]));
        __syncthreads();  // spart's place becomes dZ3
        const float inv = 1.f / s;
#pragma unroll 1
        for (int c = 8 * g; c < kClusters; c += 64) {
            tmem_ld8x2(tl + (uint32_t)c, tl + (uint32_t)c + 32u, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                v[j] = quotient(v[j], s, inv);
                if (c + column_of(j) == y) {
                    loss -= __logf(fmaxf(v[j], 1e-30f));
                    right += am == y ? 1.f : 0.f;
                    v[j] -= 1.f;
                }
                v[j] *= scale;
            }
            put_group(sG, r, c, kClusters, v);
            put_group(sG, r, c + 32, kClusters, v + 8);
            const float sum = column_sums(v, lane);
            if (!(lane & 1)) scol[q * kClusters + c + column_of(lane >> 1)] = sum;
        }
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kClusters / 16; ++ks)  // dH2 = dZ3 W3
                tc_mma(tbase, along_cols(sG, kClusters, ks), along_rows(sW3, kHidden, ks), idesc_bf16(kTile, kHidden) | kBT, ks > 0);
            tc_commit(bar);
            for (int h = 0; h < 2; ++h)  // dW3 += dZ3^T H2, behind it
                for (int ks = 0; ks < kTile / 16; ++ks)
                    tc_mma(tbase + 256 + 64 * h, along_rows(sG, kClusters, ks, 128 * h), along_rows(sH2, kHidden, ks),
                           idesc_bf16(128, kHidden) | kAT | kBT, acc | (ks > 0));
        }
        if (threadIdx.x < kClusters)
            gb3 += (scol[threadIdx.x] + scol[kClusters + threadIdx.x]) +
                   (scol[2 * kClusters + threadIdx.x] + scol[3 * kClusters + threadIdx.x]);
        if (!(ok = await())) break;
        tmem_ld16(tl + 16u * g, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = (live2 >> j & 1u) ? v[j] : 0.f;
        put_group(sD, r, 16 * g, kDCols, v);
        put_group(sD, r, 16 * g + 8, kDCols, v + 8);
        const float sum2 = column_sums(v, lane);
        if (!(lane & 1)) scol2[q * kHidden + 16 * g + (lane >> 1)] = sum2;
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kHidden / 16; ++ks)  // dH1 = dZ2 W2
                tc_mma(tbase + 64, along_cols(sD, kDCols, ks), along_rows(sW2, kHidden, ks), idesc_bf16(kTile, kHidden) | kBT, ks > 0);
            tc_commit(bar);
        }
        if (!(ok = await())) break;
        tmem_ld16(tl + 64u + 16u * g, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = (live1 >> j & 1u) ? v[j] : 0.f;
        put_group(sD, r, kHidden + 16 * g, kDCols, v);
        put_group(sD, r, kHidden + 16 * g + 8, kDCols, v + 8);
        const float sum1 = column_sums(v, lane);
        if (!(lane & 1)) scol1[q * kHidden + 16 * g + (lane >> 1)] = sum1;
        publish();
        if (threadIdx.x == 0) {
            for (int ks = 0; ks < kTile / 16; ++ks) {
                // [dZ2 | dZ1]^T H1 (its first half is dW2) and X^T dZ1
                tc_mma(tbase + 384, along_rows(sD, kDCols, ks), along_rows(sH1, kHidden, ks), idesc_bf16(128, kHidden) | kAT | kBT,
                       acc | (ks > 0));
                tc_mma(tbase + 448, along_rows(sX, kXCols, ks), along_rows(sD, kDCols, ks, kHidden),
                       idesc_bf16(128, kHidden) | kAT | kBT, acc | (ks > 0));
            }
            tc_commit(bar);
        }
        if (threadIdx.x < 2 * kHidden) {
            const float* sc = (threadIdx.x < kHidden ? scol1 : scol2) + (threadIdx.x & (kHidden - 1));
            gb21 += (sc[0] + sc[kHidden]) + (sc[2 * kHidden] + sc[3 * kHidden]);
        }
        // the gradients are done with this tile's operands before the next
        if (!(ok = await())) break;
        acc = 1;
    }
    if (ok) {
        float* out = part + (size_t)blockIdx.x * kPartFloats;
        float v[16];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            tmem_ld16(tl + 256u + 64u * h + 16u * g, v);
            float4* w = (float4*)(out + kOffW3 + (h * 128 + r) * kHidden + 16 * g);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        tmem_ld16(tl + 384u + 16u * g, v);
        if (r < kHidden) {
            float4* w = (float4*)(out + kOffW2 + r * kHidden + 16 * g);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        tmem_ld16(tl + 448u + 16u * g, v);
        if (r < kFeat)
#pragma unroll
            for (int j = 0; j < 16; ++j) out[kOffW1 + (16 * g + j) * kFeat + r] = v[j];
        if (threadIdx.x < kClusters) out[kOffB3 + threadIdx.x] = gb3;
        if (threadIdx.x < kHidden) out[kOffB1 + threadIdx.x] = gb21;
        else if (threadIdx.x < 2 * kHidden) out[kOffB2 + threadIdx.x - kHidden] = gb21;
        for (int off = 16; off; off >>= 1) {
            loss += __shfl_xor_sync(0xffffffffu, loss, off);
            right += __shfl_xor_sync(0xffffffffu, right, off);
        }
        __syncthreads();  // scol's last column sums are read
        if (lane == 0) {
            sred[warp] = loss;
            sred[16 + warp] = right;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            float t = 0.f;
            for (int w = 0; w < kTrainThreads / 32; ++w) t += sred[16 * threadIdx.x + w];
            out[kParams + threadIdx.x] = t;
        }
    } else if (threadIdx.x == 0) {
        // MMAs in flight get one more bounded window before TMEM is released:
        // those of the wait that failed, then those issued behind it
        if (mbar_wait_bounded(bar, phase ^ 1u, status)) {
            tc_commit(bar);
            mbar_wait_bounded(bar, phase, status);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tbase, 512);
}

// Sums the partial gradients in CTA order, then either stores them (grads)
// or takes the SGD step with momentum on the FP32 parameters and refreshes
// the BF16 weights.  W1's columns past the 105 features are padding: never
// updated, zero in BF16.  Eight partials in flight per thread hide the L2
// latency of the 64 that 8,192 records leave.
__global__ void __launch_bounds__(256)
    apply_kernel(const float* part, int nparts, float* P, float* V, uint16_t* Wb, float* grads, float* acc, float lr, float mom) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    grid_dependency_wait_and_release();
    if (i >= kParams + 2) return;
    float s = 0.f;
    int k = 0;
    for (; k + 8 <= nparts; k += 8) {
        float t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = load_written(part + (size_t)(k + j) * kPartFloats + i);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += t[j];
    }
    for (; k < nparts; ++k) s += load_written(part + (size_t)k * kPartFloats + i);
    if (i >= kParams) {
        acc[i - kParams] = s;
        return;
    }
    if (grads) {
        grads[i] = s;
        return;
    }
    if (i < kOffB1 && i % kFeat >= 105) {
        Wb[i] = 0;
        return;
    }
    const float v = mom * load_written(V + i) + s;
    V[i] = v;
    const float w = load_written(P + i) - lr * v;
    P[i] = w;
    Wb[i] = f2bf(w);
}

}  // namespace

int train_step(pbg_scene* s, Learner* L, const uint16_t* X, const int32_t* Y, int B, bool update, bool chained,
               cudaStream_t st) {
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const int tiles = B / kTile;
    const int ctas = std::min(tiles, sms);
    int rc;
    if ((rc = ensure(L->part, (size_t)ctas * kPartFloats * 4)) || (rc = ensure(L->acc, 64))) return rc;
    if (!update && (rc = ensure(L->G, (size_t)kParams * 4))) return rc;
    // a per-device setting (cheap, idempotent): set on every call so that each
    // device the library launches on has it
    PBG_CUDA(cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.stream = st;
    cfg.attrs = &overlap;
    cfg.numAttrs = chained ? 1 : 0;  // the records may still be on their way to a call's first step
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kTrainThreads);
    cfg.dynamicSmemBytes = kTrainSmem;
    PBG_CUDA(cudaLaunchKernelEx(&cfg, train_kernel, X, Y, tiles, (const uint16_t*)L->Wb.ptr, (const float*)L->P.ptr,
                                1.f / (float)B, (float*)L->part.ptr, (int*)s->err.ptr));
    cfg.gridDim = dim3((kParams + 2 + 255) / 256);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.numAttrs = 1;
    PBG_CUDA(cudaLaunchKernelEx(&cfg, apply_kernel, (const float*)L->part.ptr, ctas, (float*)L->P.ptr, (float*)L->V.ptr,
                                (uint16_t*)L->Wb.ptr, update ? (float*)nullptr : (float*)L->G.ptr, (float*)L->acc.ptr, L->lr,
                                L->momentum));
    s->counters.kernel_launches += 2;
    return PBG_OK;
}

}  // namespace pbg
