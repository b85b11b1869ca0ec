// k_sort.cu -- bounding box, Morton codes, LSD radix sort and the sorted gather.
//
// Stage 1-2 of the step (reference: BarnesHutCuda.cu:648-711).  The box is
// reduced in one launch (last-block-done) and squared on the device, so the
// step never returns to the host; Morton codes are bit-exact with CU:54-69;
// the sort is a project-written stable LSD radix sort over all 64 key bits,
// so its order equals cub::DeviceRadixSort::SortPairs at CU:692 (any stable
// sort of (code, current index) gives the same permutation).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "nb_internal.cuh"

namespace cg = cooperative_groups;

namespace nb {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBoxThreads = 512;
constexpr double kBoxSeed = 1.7976931348623157e308;  // DBL_MAX

__device__ __forceinline__ double warp_min(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// This step's radix passes (the top bytes of the key the sort orders by), from
// the histogram of the last tree.  Without `adaptive` (or with a forced count)
// no histogram is used.  One warp.
__device__ __forceinline__ int sort_passes_of(const DeviceScalars* s, int64_t n, int adaptive) {
    const int forced = s->sort_passes_forced;
    if (forced > 0) return min(forced, 8);
    return adaptive ? choose_sort_passes(s->lcp_hist, n) : 8;
}

// Consumes the histogram and resets what the later kernels of a step count in,
// and in a new step the interaction counters.  One warp.
__device__ __forceinline__ void start_sort(DeviceScalars* s, int passes, int new_step) {
    const int lane = threadIdx.x & 31;
    s->lcp_hist[lane] = 0;
    if (lane != 0) return;
    s->sort_passes = passes;
    s->lcp_hist[32] = 0;
    s->tie_count[0] = 0;
    s->tie_count[1] = 0;
    s->group_ticket = 0;
    if (new_step) {
        s->cell_terms = 0;
        s->body_terms = 0;
        s->stack_hw = 0;
    }
}

// Exact FP64 min/max of all positions, reduced per block, then folded and
// squared by the last block to finish (CU:78-114 + the host squaring at
// CU:665-677, done here on the device in the same FP64 operations).  Min and
// max are exact in any order, so the reduction tree is free: each thread
// keeps four loads in flight, and the last block folds the partials with all
// its threads.
__device__ __forceinline__ void box_fold(double& xmin, double& xmax, double& ymin, double& ymax,
                                         double (*red)[kBoxThreads / 32]) {
    xmin = warp_min(xmin);
    xmax = warp_max(xmax);
    ymin = warp_min(ymin);
    ymax = warp_max(ymax);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        red[0][warp] = xmin;
        red[1][warp] = xmax;
        red[2][warp] = ymin;
        red[3][warp] = ymax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kBoxThreads / 32; ++w) {
            xmin = fmin(xmin, red[0][w]);
            xmax = fmax(xmax, red[1][w]);
            ymin = fmin(ymin, red[2][w]);
            ymax = fmax(ymax, red[3][w]);
        }
    }
}

// The squared root box of the extremes (host squaring, CU:665-677) and the
// Morton kernel's scale factors (CU:122-123).
struct RootBox {
    double x0, x1, y0, y1, inv_w, inv_h;
};
__device__ __forceinline__ RootBox square_box(double bx0, double bx1, double by0, double by1) {
    const double x_range = bx1 - bx0;
    const double y_range = by1 - by0;
    if (x_range > y_range) {
        const double mid = (by0 + by1) * 0.5;
        by0 = mid - x_range * 0.5;
        by1 = mid + x_range * 0.5;
    } else {
        const double mid = (bx0 + bx1) * 0.5;
        bx0 = mid - y_range * 0.5;
        bx1 = mid + y_range * 0.5;
    }
    return {bx0, bx1, by0, by1, 1.0 / (bx1 - bx0), 1.0 / (by1 - by0)};
}
__device__ __forceinline__ void write_box(DeviceScalars* s, const RootBox& b) {
    s->box[0] = b.x0;
    s->box[1] = b.x1;
    s->box[2] = b.y0;
    s->box[3] = b.y1;
    s->center[0] = 0.5 * (b.x0 + b.x1);
    s->center[1] = 0.5 * (b.y0 + b.y1);
    s->inv_wh[0] = b.inv_w;
    s->inv_wh[1] = b.inv_h;
    // CU:717 root width_sq, then CU:216 child_wsq = parent * 0.25 per level.
    const double w = b.x1 - b.x0;
    double wsq = w * w;
    for (int l = 0; l <= kMaxLevel; ++l) {
        s->wsq[l] = wsq;
        wsq *= 0.25;
    }
}

__global__ void __launch_bounds__(kBoxThreads)
bbox_kernel(const double2* pos, int64_t n, double* partials,
            DeviceScalars* s, int adaptive, int new_step, unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    double xmin = INFINITY, xmax = -INFINITY, ymin = INFINITY, ymax = -INFINITY;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {
        double2 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = pos[i + u * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            xmin = fmin(xmin, p[u].x);
            xmax = fmax(xmax, p[u].x);
            ymin = fmin(ymin, p[u].y);
            ymax = fmax(ymax, p[u].y);
        }
    }
    for (; i < n; i += stride) {
        const double2 p = pos[i];
        xmin = fmin(xmin, p.x);
        xmax = fmax(xmax, p.x);
        ymin = fmin(ymin, p.y);
        ymax = fmax(ymax, p.y);
    }
    __shared__ double red[4][kBoxThreads / 32];
    __shared__ bool last_block;
    box_fold(xmin, xmax, ymin, ymax, red);
    if (threadIdx.x == 0) {
        double* out = partials + 4 * blockIdx.x;
        out[0] = xmin;
        out[1] = xmax;
        out[2] = ymin;
        out[3] = ymax;
        __threadfence();
        last_block = atomicAdd(&s->bbox_ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    // CU:649-654 seeds with +-DBL_MAX; folding from there is identical.
    double bx0 = kBoxSeed, bx1 = -kBoxSeed, by0 = kBoxSeed, by1 = -kBoxSeed;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
        const double* in = partials + 4 * b;
        bx0 = fmin(bx0, __ldcg(in + 0));
        bx1 = fmax(bx1, __ldcg(in + 1));
        by0 = fmin(by0, __ldcg(in + 2));
        by1 = fmax(by1, __ldcg(in + 3));
    }
    __syncthreads();  // red[] is reused
    box_fold(bx0, bx1, by0, by1, red);
    if (threadIdx.x < 32) {
        const int passes = sort_passes_of(s, n, adaptive);
        __syncwarp();
        start_sort(s, passes, new_step);
    }
    if (threadIdx.x == 0) {
        write_box(s, square_box(bx0, bx1, by0, by1));
        s->bbox_ticket = 0;
    }
}

__device__ __forceinline__ uint64_t expand_bits_2d(uint32_t v) {
    uint64_t x = v;
    x = (x | (x << 16)) & 0x0000FFFF0000FFFFull;
    x = (x | (x << 8)) & 0x00FF00FF00FF00FFull;
    x = (x | (x << 4)) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | (x << 2)) & 0x3333333333333333ull;
    x = (x | (x << 1)) & 0x5555555555555555ull;
    return x;
}

// What the onesweep passes count in: the digit histograms, the tile counters
// and the status words of the passes that will run.  The Morton pass resets it.
struct SortState {
    uint32_t* hist = nullptr;     // nullptr: no onesweep passes follow
    unsigned* tile_counter = nullptr;
    uint32_t* status = nullptr;
    int tiles = 0;
};

__device__ __forceinline__ void reset_sort(const SortState& z, int passes) {
    if (!z.hist) return;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x, per_pass = 256 * (int64_t)sort_status_rows(z.tiles);
    for (int64_t k = t0; k < 8 * 256; k += step) z.hist[k] = 0;
    if (t0 < 8) z.tile_counter[t0] = 0;
    for (int64_t k = (8 - passes) * per_pass + t0; k < 8 * per_pass; k += step) z.status[k] = 0;
}

__device__ __forceinline__ uint64_t morton_code(double2 p, double x0, double y0, double inv_w,
                                                double inv_h) {
    const double nx = (p.x - x0) * inv_w;
    const double ny = (p.y - y0) * inv_h;
    const uint32_t ix = __double2uint_rd(fmin(fmax(nx * 4294967296.0, 0.0), 4294967295.0));
    const uint32_t iy = __double2uint_rd(fmin(fmax(ny * 4294967296.0, 0.0), 4294967295.0));
    return (expand_bits_2d(ix) << 1) | expand_bits_2d(iy);
}

// CU:117-132: code from (p - min) * (1 / width), quantised to 32 bits per axis
// with round-down; x bits land on odd positions.  val = current slot.  The
// codes go to the buffer the first radix pass reads: pass k reads buffer
// k & 1, and the first of the step's sort_passes passes is 8 - sort_passes,
// so the last one always writes buffer 0.
__global__ void morton_kernel(const double2* pos, int64_t n,
                              const DeviceScalars* s, uint64_t* key0,
                              uint64_t* key1, uint32_t* val0,
                              uint32_t* val1, SortState z) {
    chain_begin();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int passes = s->sort_passes;
    const double2 p = i < n ? pos[i] : make_double2(0.0, 0.0);
    const uint64_t code = morton_code(p, s->box[0], s->box[2], s->inv_wh[0], s->inv_wh[1]);
    reset_sort(z, passes);
    if (i >= n) return;
    const bool odd = passes & 1;
    (odd ? key1 : key0)[i] = code;
    (odd ? val1 : val0)[i] = (uint32_t)i;
}

// ---------------------------------------------------------------------------
// Batched universes: per-universe boxes and 54-bit Morton codes under the
// universe id.  Doubles are reduced through an order-preserving integer image
// so plain 64-bit atomicMin/atomicMax give the exact FP64 min/max.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ordered_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_ordered(unsigned long long o) {
    const unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    return __longlong_as_double((long long)b);
}

// A warp takes kBoxRows rows of 32 consecutive bodies and folds a universe's
// extremes in registers until its bodies end: one set of four atomics per warp
// and universe.  (One per row, contending for 256 words: boxes and codes of 64
// universes, 3.4M bodies, took 132 us, now 56.)
constexpr int kBoxRows = 16;

__global__ void __launch_bounds__(256)
bbox_batch_kernel(const double2* pos, int64_t n, Batch b, unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    const int lane = threadIdx.x & 31;
    const int64_t base =
        ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32 * kBoxRows + lane;
    int current = -1;  // the universe being folded (warp-uniform), -1: none
    double x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
    auto put = [&](int u, double xmin, double xmax, double ymin, double ymax) {
        // min-encoded: a maximum through the complement
        atomicMin(b.boxbits + 4 * u, ordered_bits(xmin));
        atomicMin(b.boxbits + 4 * u + 1, ~ordered_bits(xmax));
        atomicMin(b.boxbits + 4 * u + 2, ordered_bits(ymin));
        atomicMin(b.boxbits + 4 * u + 3, ~ordered_bits(ymax));
    };
    auto flush = [&] {
        if (current < 0) return;
        const double a = warp_min(x0), c = warp_max(x1), d = warp_min(y0), f = warp_max(y1);
        if (lane == 0) put(current, a, c, d, f);
        x0 = y0 = INFINITY;
        x1 = y1 = -INFINITY;
    };
#pragma unroll 4
    for (int r = 0; r < kBoxRows; ++r) {
        const int64_t i = base + 32 * r;
        const bool valid = i < n;
        const int u = valid ? b.uid[i] : -1;
        const double2 p = valid ? pos[i] : make_double2(0.0, 0.0);
        const int u0 = __shfl_sync(kFull, u, 0);
        if (u0 < 0) break;  // past the last body
        if (u0 != current) {
            flush();
            current = u0;
        }
        if (u == u0) {
            x0 = fmin(x0, p.x);
            x1 = fmax(x1, p.x);
            y0 = fmin(y0, p.y);
            y1 = fmax(y1, p.y);
        } else if (valid) {  // the row's next universes: body by body
            put(u, p.x, p.x, p.y, p.y);
        }
    }
    flush();
}

// Squares every universe's box as the single-universe path does, and resets
// the reduction slots for the next step.
__global__ void bbox_batch_finish(Batch b, DeviceScalars* s, int64_t n,
                                  int new_step) {
    chain_begin();
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u < 32) {
        const int passes = sort_passes_of(s, n, 1);
        __syncwarp();
        start_sort(s, passes, new_step);
    }
    if (u >= b.nuni) return;
    unsigned long long* e = b.boxbits + 4 * u;
    double x0 = from_ordered(e[0]), x1 = from_ordered(~e[1]);
    double y0 = from_ordered(e[2]), y1 = from_ordered(~e[3]);
    const double x_range = x1 - x0, y_range = y1 - y0;
    if (x_range > y_range) {
        const double mid = (y0 + y1) * 0.5;
        y0 = mid - x_range * 0.5;
        y1 = mid + x_range * 0.5;
    } else {
        const double mid = (x0 + x1) * 0.5;
        x0 = mid - y_range * 0.5;
        x1 = mid + y_range * 0.5;
    }
    const double w = x1 - x0;
    b.lo[u] = make_double2(x0, y0);
    b.center[u] = make_double2(0.5 * (x0 + x1), 0.5 * (y0 + y1));
    const double w2 = w > 0.0 ? w * w : 1.0;  // a one-point universe: any width
    b.w2[u] = w2;
    b.inv_w[u] = 1.0 / sqrt(w2);
    e[0] = ~0ull;
    e[1] = ~0ull;
    e[2] = ~0ull;
    e[3] = ~0ull;
}

__global__ void morton_batch_kernel(const double2* pos, int64_t n, Batch b,
                                    const DeviceScalars* s,
                                    uint64_t* key0, uint64_t* key1,
                                    uint32_t* val0, uint32_t* val1,
                                    SortState z) {
    chain_begin();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int passes = s->sort_passes;
    if (i >= n) {
        reset_sort(z, passes);
        return;
    }
    const int u = b.uid[i];
    const double2 lo = b.lo[u];
    const double inv_w = b.inv_w[u];
    const double2 p = pos[i];
    reset_sort(z, passes);
    // (cluster sorts read buffer 0)
    const bool odd = z.hist && (passes & 1);
    uint64_t* key = odd ? key1 : key0;
    uint32_t* val = odd ? val1 : val0;
    const double scale = (double)(1u << kBatchMortonBits);
    const double top = scale - 1.0;
    const uint32_t ix = __double2uint_rd(fmin(fmax((p.x - lo.x) * inv_w * scale, 0.0), top));
    const uint32_t iy = __double2uint_rd(fmin(fmax((p.y - lo.y) * inv_w * scale, 0.0), top));
    key[i] = ((uint64_t)u << (2 * kBatchMortonBits)) | (expand_bits_2d(ix) << 1) | expand_bits_2d(iy);
    val[i] = (uint32_t)i;
}

// ---------------------------------------------------------------------------
// LSD radix sorts with 8-bit digits: inside clusters of blocks up to
// kClusterSortMax keys, by onesweep passes over global memory above.
// ---------------------------------------------------------------------------
constexpr int kWarps = kSortThreads / 32;

// Exclusive scan of one value per thread over a 256-thread block.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_tot,
                                                         uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kWarps ? warp_tot[lane] : 0;
        uint32_t winc = w;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, winc, o);
            if (lane >= o) winc += t;
        }
        if (lane < kWarps) warp_tot[lane] = winc - w;
        if (lane == kWarps - 1 && total) *total = winc;
    }
    __syncthreads();
    const uint32_t r = warp_tot[warp] + inc - v;
    __syncthreads();
    return r;
}

// Lanes holding the same 8-bit digit, from eight ballots (the ballot path
// keeps this off the pipe that serialises __match_any_sync).
__device__ __forceinline__ unsigned digit_peers(uint32_t d, bool valid) {
    unsigned peers = __ballot_sync(kFull, valid);
    if (!valid) peers = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const unsigned m = __ballot_sync(kFull, bit);
        peers &= bit ? m : ~m;
    }
    return valid ? peers : (1u << (threadIdx.x & 31));
}

// ---------------------------------------------------------------------------
// Cluster sort, up to kClusterSortMax keys.  There a pass over global memory is
// a chain of latencies (7 us a pass at 16,384 keys), so one cluster of up to 16
// blocks keeps all keys in shared memory and scatters them between its blocks'
// shared memories, with one cluster barrier after the digit counts and one
// after the scatter.  Box, codes and passes are one kernel.  Same order as the
// onesweep passes: by the top sort_passes bytes, equal ones in input order.
// Box to sorted keys, us, with onesweep passes and so: 1,001 bodies 37 and 16,
// 16,384 49 and 32, 32,768 60 and 44.  With four keys a thread (65,536) a pass
// takes as long as over global memory; sorting chunks by several clusters and
// merging them took longer (262,144 bodies 69 and 78).
// ---------------------------------------------------------------------------
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterMost = 16;  // blocks in a cluster
static_assert(kClusterSortMax == 2 * kClusterMost * kClusterThreads, "at most two keys per thread");

// Where the codes come from: the bodies (box and codes are made here), or
// key_in (batched universes, whose codes have been made).
enum { kSrcBodies, kSrcKeys };

template <int kItems>
struct ClusterSmem {
    uint64_t key[kClusterThreads * kItems];  // written by the whole cluster
    uint32_t val[kClusterThreads * kItems];
    uint64_t own_key[kClusterThreads * kItems];  // this block's keys by digit
    uint32_t own_val[kClusterThreads * kItems];
    uint16_t whist[kClusterWarps][256];  // per warp, then exclusive within its part
    uint32_t match[kClusterWarps][256];  // per warp and digit: the row's lanes with it
    uint32_t count[256];                 // this block's digits, read by the whole cluster
    uint32_t before[4][256], total[4][256];
    uint32_t off[4][256];                // place of a part's keys among the block's
    uint32_t base[256];                  // place in the cluster less place in the block
    uint32_t warp_tot[2][8];
    double red[4][kClusterWarps];
    double box[4];                       // this block's extremes, read by the whole cluster
    int passes;
};

// Rank of this lane's digit d in the warp's keys so far, row by row: the lanes
// of the row with the same digit set their bits in the digit's word of match[]
// (all zero between rows), whist[] counts the rows before.
__device__ __forceinline__ uint32_t row_rank(uint32_t* match, uint16_t* whist, uint32_t d,
                                             bool valid, unsigned below) {
    if (valid) atomicOr(&match[d], 1u << (threadIdx.x & 31));
    __syncwarp();
    const unsigned peers = valid ? match[d] : 0u;
    const uint32_t b = valid ? whist[d] : 0u;
    __syncwarp();
    if (valid && (peers & below) == 0) {
        whist[d] = (uint16_t)(b + __popc(peers));
        match[d] = 0;
    }
    __syncwarp();
    return b + __popc(peers & below);
}

// Inclusive scan over the threads of each of the first eight warps; their totals.
__device__ __forceinline__ uint32_t digit_scan(uint32_t v, uint32_t* warp_tot) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tot[threadIdx.x >> 5] = v;
    return v;
}

// The two halves of a cluster barrier: what a thread wrote before it arrives
// is visible to the cluster's threads that have waited.
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int kItems, int kSrc>
__global__ void __launch_bounds__(kClusterThreads, 1)
cluster_sort(const double2* pos, int64_t n, DeviceScalars* s, int adaptive,
             int new_step, int fixed_passes, const uint64_t* key_in, uint64_t* key_out,
             uint32_t* val_out, unsigned long long* mark0, unsigned long long* mark1) {
    chain_begin();
    mark_start(mark0);
    constexpr int kTile = kClusterThreads * kItems;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem<kItems>& S = *reinterpret_cast<ClusterSmem<kItems>*>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const int me = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = tid >> 8, digit = tid & 255;
    // a warp's keys: kItems rows of 32; slots from n on (the last chunk's end) stay empty
    const int slot0 = warp * 32 * kItems + lane;
    const int64_t first = (int64_t)blockIdx.x * kTile + slot0;
    uint64_t k_reg[kItems];
    uint32_t v_reg[kItems], r_reg[kItems];
    int passes = fixed_passes;
    if (kSrc == kSrcKeys) {
#pragma unroll
        for (int k = 0; k < kItems; ++k) k_reg[k] = first + 32 * k < n ? key_in[first + 32 * k] : 0ull;
        if (passes == 0) passes = s->sort_passes;
    } else {
        double2 p[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            p[k] = first + 32 * k < n ? pos[first + 32 * k] : make_double2(0.0, 0.0);
        RootBox box;
        {
            // (CU:649-654 seeds with +-DBL_MAX, which show where an axis has no
            // finite value: nb_morton_sort_static takes any positions)
            double v[4] = {kBoxSeed, -kBoxSeed, kBoxSeed, -kBoxSeed};
#pragma unroll
            for (int k = 0; k < kItems; ++k)
                if (first + 32 * k < n) {
                    v[0] = fmin(v[0], p[k].x);
                    v[1] = fmax(v[1], p[k].x);
                    v[2] = fmin(v[2], p[k].y);
                    v[3] = fmax(v[3], p[k].y);
                }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                v[q] = (q & 1) ? warp_max(v[q]) : warp_min(v[q]);
                if (lane == 0) S.red[q][warp] = v[q];
            }
            __syncthreads();
            if (warp < 4) {  // warp q folds extreme q
                const double x = S.red[warp][lane];
                const double f = (warp & 1) ? warp_max(x) : warp_min(x);
                if (lane == 0) S.box[warp] = f;
            } else if (warp == 4) {
                const int chosen = fixed_passes ? fixed_passes : sort_passes_of(s, n, adaptive);
                if (lane == 0) S.passes = chosen;
            }
            cluster.sync();
            double m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double x = cluster.map_shared_rank(S.box, min(lane, blocks - 1))[q];
                m[q] = (q & 1) ? warp_max(x) : warp_min(x);
            }
            box = square_box(m[0], m[1], m[2], m[3]);
            passes = S.passes;
            if (me == 0 && warp == 0) {  // the cluster has read the histogram
                start_sort(s, passes, new_step);
                if (lane == 0) write_box(s, box);
            }
        }
#pragma unroll
        for (int k = 0; k < kItems; ++k) k_reg[k] = morton_code(p[k], box.x0, box.y0, box.inv_w, box.inv_h);
    }
    mark_start(mark1);
#pragma unroll
    for (int k = 0; k < kItems; ++k) v_reg[k] = (uint32_t)(first + 32 * k);
    const unsigned below = lanemask_lt();
    const int held = (int)max((int64_t)0, min((int64_t)kTile, n - (int64_t)blockIdx.x * kTile));
#pragma unroll
    for (int k = lane; k < 256; k += 32) S.match[warp][k] = 0;
    for (int pass = 8 - passes; pass < 8; ++pass) {
#pragma unroll
        for (int k = lane; k < 128; k += 32) reinterpret_cast<uint32_t*>(S.whist[warp])[k] = 0;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            r_reg[k] = row_rank(S.match[warp], S.whist[warp], (uint32_t)(k_reg[k] >> (8 * pass)) & 255u,
                                first + 32 * k < n, below);
        __syncthreads();
        {   // exclusive over the part's warps
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kClusterWarps / 4; ++w) {
                const uint32_t c = S.whist[part * (kClusterWarps / 4) + w][digit];
                S.whist[part * (kClusterWarps / 4) + w][digit] = (uint16_t)run;
                run += c;
            }
            S.off[part][digit] = run;
        }
        __syncthreads();
        // places in the block: exclusive scan of its digit counts
        uint32_t count = 0, inc = 0, mine = 0;
        if (tid < 256) {
            count = S.off[0][tid] + S.off[1][tid] + S.off[2][tid] + S.off[3][tid];
            S.count[tid] = count;
            inc = digit_scan(count, S.warp_tot[0]);
        }
        cluster_arrive();  // (the counts)
        __syncthreads();
        if (tid < 256) {
            mine = inc - count;
            for (int w = 0; w < warp; ++w) mine += S.warp_tot[0][w];
            uint32_t off = mine;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t c = S.off[p][tid];
                S.off[p][tid] = off;
                off += c;
            }
        }
        __syncthreads();
        // the block's keys by digit, so that they leave in runs
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (first + 32 * k >= n) continue;
            const uint32_t d = (uint32_t)(k_reg[k] >> (8 * pass)) & 255u;
            const uint32_t at = S.off[part][d] + S.whist[warp][d] + r_reg[k];
            S.own_key[at] = k_reg[k];
            S.own_val[at] = v_reg[k];
        }
        cluster_wait();  // every block's counts are there, and its keys in registers
        {   // this digit in a quarter of the blocks: before this block, and in all
            uint32_t before = 0, total = 0;
            for (int c = part; c < blocks; c += 4) {
                const uint32_t x = cluster.map_shared_rank(S.count, c)[digit];
                total += x;
                before += c < me ? x : 0u;
            }
            S.before[part][digit] = before;
            S.total[part][digit] = total;
        }
        __syncthreads();
        if (tid < 256) {  // the digits' bases: exclusive scan of their totals
            count = S.total[0][tid] + S.total[1][tid] + S.total[2][tid] + S.total[3][tid];
            inc = digit_scan(count, S.warp_tot[1]);
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t off = inc - count - mine;
            for (int w = 0; w < warp; ++w) off += S.warp_tot[1][w];
#pragma unroll
            for (int p = 0; p < 4; ++p) off += S.before[p][tid];
            S.base[tid] = off;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int j = k * kClusterThreads + tid;
            if (j >= held) continue;
            const uint64_t key = S.own_key[j];
            const uint32_t at = S.base[(uint32_t)(key >> (8 * pass)) & 255u] + (uint32_t)j;
            cluster.map_shared_rank(S.key, at / kTile)[at % kTile] = key;
            cluster.map_shared_rank(S.val, at / kTile)[at % kTile] = S.own_val[j];
        }
        cluster.sync();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            k_reg[k] = S.key[slot0 + 32 * k];
            v_reg[k] = S.val[slot0 + 32 * k];
        }
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (first + 32 * k < n) {
            key_out[first + 32 * k] = k_reg[k];
            val_out[first + 32 * k] = v_reg[k];
        }
}

// ---------------------------------------------------------------------------
// Counting passes (nb_morton_sort_static above kClusterSortMax keys): one
// kernel counts each tile's digits, the next adds up the counts of the tiles
// before its own and scatters.  No block waits on another, so the stage needs
// no error word, which that entry point could not report.
// ---------------------------------------------------------------------------
constexpr int kCountThreads = 1024;
constexpr int kCountItems = kCountTile / kCountThreads;
constexpr int kCountWarps = kCountThreads / 32;

__global__ void __launch_bounds__(kCountThreads)
count_digits(const uint64_t* key, int64_t n, int pass, uint16_t* counts) {
    chain_begin();
    __shared__ uint32_t hist[4][256];  // one per quarter of the block
    const int tid = threadIdx.x, part = tid >> 8;
    hist[part][tid & 255] = 0;
    const int64_t base = (int64_t)blockIdx.x * kCountTile + tid;
    uint64_t k[kCountItems];
#pragma unroll
    for (int q = 0; q < kCountItems; ++q)
        k[q] = base + q * kCountThreads < n ? key[base + q * kCountThreads] : 0ull;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kCountItems; ++q)
        if (base + q * kCountThreads < n)
            atomicAdd(&hist[part][(uint32_t)(k[q] >> (8 * pass)) & 255u], 1u);
    __syncthreads();
    if (tid < 256)
        counts[(int64_t)blockIdx.x * 256 + tid] =
            (uint16_t)(hist[0][tid] + hist[1][tid] + hist[2][tid] + hist[3][tid]);
}

__global__ void __launch_bounds__(kCountThreads, 1)
count_scatter(const uint64_t* key_in, const uint32_t* val_in,
              uint64_t* key_out, uint32_t* val_out, int64_t n, int pass,
              const uint16_t* counts, int tiles) {
    chain_begin();
    __shared__ uint16_t whist[kCountWarps][256];  // per warp, then exclusive within its part
    __shared__ uint32_t match[kCountWarps][256];  // per warp and digit: the row's lanes with it
    // after the ranking, in match[]'s place (48 KB of static shared memory)
    auto* before = reinterpret_cast<uint32_t(*)[256]>(&match[0][0]);
    auto* total = reinterpret_cast<uint32_t(*)[256]>(&match[8][0]);
    auto* off = reinterpret_cast<uint32_t(*)[256]>(&match[16][0]);
    uint32_t* warp_tot = &match[20][0];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x, part = tid >> 8, digit = tid & 255;
    // a warp's keys: kCountItems rows of 32
    const int64_t first = (int64_t)tile * kCountTile + warp * (32 * kCountItems) + lane;
    uint64_t k_reg[kCountItems];
    uint32_t v_reg[kCountItems], r_reg[kCountItems];
#pragma unroll
    for (int k = 0; k < kCountItems; ++k) {
        const bool valid = first + 32 * k < n;
        k_reg[k] = valid ? key_in[first + 32 * k] : 0ull;
        v_reg[k] = valid ? val_in[first + 32 * k] : 0u;
    }
    // two digits in an eighth of the tiles: before this tile, and in all
    uint32_t lo_before = 0, hi_before = 0, lo_all = 0, hi_all = 0;
    {
        const uint32_t* pairs = reinterpret_cast<const uint32_t*>(counts) + (tid & 127);
#pragma unroll 8
        for (int q = tid >> 7; q < tiles; q += 8) {
            const uint32_t x = pairs[q * 128], lo = x & 0xffffu, hi = x >> 16;
            lo_all += lo;
            hi_all += hi;
            lo_before += q < tile ? lo : 0u;
            hi_before += q < tile ? hi : 0u;
        }
    }
#pragma unroll
    for (int k = lane; k < 128; k += 32) reinterpret_cast<uint32_t*>(whist[warp])[k] = 0;
#pragma unroll
    for (int k = lane; k < 256; k += 32) match[warp][k] = 0;
    __syncwarp();
    const unsigned below = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kCountItems; ++k)
        r_reg[k] = row_rank(match[warp], whist[warp], (uint32_t)(k_reg[k] >> (8 * pass)) & 255u,
                            first + 32 * k < n, below);
    __syncthreads();
    before[tid >> 7][2 * (tid & 127)] = lo_before;
    before[tid >> 7][2 * (tid & 127) + 1] = hi_before;
    total[tid >> 7][2 * (tid & 127)] = lo_all;
    total[tid >> 7][2 * (tid & 127) + 1] = hi_all;
    {   // exclusive over the part's warps
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kCountWarps / 4; ++w) {
            const uint32_t c = whist[part * (kCountWarps / 4) + w][digit];
            whist[part * (kCountWarps / 4) + w][digit] = (uint16_t)run;
            run += c;
        }
        off[part][digit] = run;
    }
    __syncthreads();
    // the digits' bases: exclusive scan of their totals
    uint32_t sum = 0, inc = 0;
    if (tid < 256) {
#pragma unroll
        for (int p = 0; p < 8; ++p) sum += total[p][tid];
        inc = digit_scan(sum, warp_tot);
    }
    __syncthreads();
    if (tid < 256) {
        uint32_t o = inc - sum;
        for (int w = 0; w < warp; ++w) o += warp_tot[w];
#pragma unroll
        for (int p = 0; p < 8; ++p) o += before[p][tid];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t c = off[p][tid];
            off[p][tid] = o;
            o += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kCountItems; ++k) {
        if (first + 32 * k >= n) continue;
        const uint32_t d = (uint32_t)(k_reg[k] >> (8 * pass)) & 255u;
        const uint32_t at = off[part][d] + whist[warp][d] + r_reg[k];
        key_out[at] = k_reg[k];
        val_out[at] = v_reg[k];
    }
}

// ---------------------------------------------------------------------------
// Onesweep LSD radix sort (the step's sort).  One pass over the keys builds
// the histograms of all eight digits; each digit pass is then a single kernel
// whose tiles learn their global offsets by decoupled look-back: a tile
// publishes its per-digit count, then sums its predecessors' counts, those of
// earlier groups of kSortGroup tiles a group at a time, until it meets a group
// whose start is known.  Tiles take their index
// from an atomic counter in the order they start, so a tile only ever waits
// on tiles that are already running.  Every wait is bounded; a wait that runs
// out sets kErrTimeout and the step reports NB_ERR_TIMEOUT.
// ---------------------------------------------------------------------------
constexpr uint32_t kFlagAgg = 1u << 31;  // a published word; the rest is the value
constexpr int kGroupBits = 20;           // a group's sum: counts below, tiles counted above
static_assert(kSortGroup * kSortItemsMax * kSortThreads < (1 << kGroupBits) && kSortGroup < 1 << (32 - kGroupBits),
              "a group's counts fit its word");
constexpr int kSpinLimit = 1 << 22;
constexpr int kLook = 4;  // words in flight (8 and 16: 4M sort 289 -> 297, 304 us)

// Histograms of the digits the radix passes sort (the top sort_passes bytes;
// the passes below return at once and need none).  A warp reads rows of 32
// consecutive keys (one coalesced load) and, per digit, finds the runs of
// equal digits in the row with one ballot: each run's first lane adds the
// run's length to the digit's bin.  The keys arrive nearly sorted (the bodies
// keep last step's order), so the high digits form long runs and most rows
// cost one shared-memory atomic per digit.
constexpr int kHistRows = 4;

__global__ void __launch_bounds__(kSortThreads)
onesweep_histogram(const uint64_t* key0, const uint64_t* key1, int64_t n,
                   const DeviceScalars* s, uint32_t* hist,
                   unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    // the Morton pass wrote the codes where the first radix pass reads them
    const uint64_t* key = (s->sort_passes & 1) ? key1 : key0;
    const int dmin = 8 - s->sort_passes;  // digits below are not sorted by a pass
    __shared__ uint32_t h[8][256];
    for (int k = threadIdx.x; k < 8 * 256; k += kSortThreads) (&h[0][0])[k] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (kSortThreads / 32);
    const int64_t w = (int64_t)blockIdx.x * (kSortThreads / 32) + (threadIdx.x >> 5);
    const unsigned after_me = ~((2u << lane) - 1u);  // lanes above this one (none for lane 31)
    // kHistRows rows per warp and iteration: their loads are in flight together
    for (int64_t row0 = w * 32 * kHistRows; row0 < n; row0 += warps * 32 * kHistRows) {
        uint64_t k[kHistRows];
#pragma unroll
        for (int r = 0; r < kHistRows; ++r) {
            const int64_t i = row0 + 32 * r + lane;
            k[r] = i < n ? key[i] : 0ull;
        }
#pragma unroll
        for (int r = 0; r < kHistRows; ++r) {
            const int64_t left = n - (row0 + 32 * r);  // valid lanes of the row are a prefix
            if (left <= 0) break;
            const int end = left < 32 ? (int)left : 32;
            const bool valid = lane < end;
            const uint64_t kp = __shfl_up_sync(kFull, k[r], 1);
            const uint64_t diff = k[r] ^ kp;
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                if (d < dmin) continue;
                const bool head = valid && (lane == 0 || ((diff >> (8 * d)) & 0xFF) != 0);
                const unsigned later = __ballot_sync(kFull, head) & after_me;
                if (head)
                    atomicAdd(&h[d][(uint32_t)(k[r] >> (8 * d)) & 0xFF],
                              (uint32_t)((later ? __ffs(later) - 1 : end) - lane));
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 8 * 256; k += kSortThreads) {
        const uint32_t v = (&h[0][0])[k];
        if (v) atomicAdd(hist + k, v);
    }
}

__device__ __forceinline__ uint32_t ld_status(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_status(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---- one-CTA bulk copies (cp.async.bulk, no multicast) into shared memory --
__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    // the barrier must be visible to the async proxy before a copy signals it
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
// bytes: a multiple of 16; both addresses 16-byte aligned
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned phase) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P1;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return done != 0;
}
// Bounded wait for phase 0 of a barrier; false if it ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar) {
    for (int k = 0; k < kSpinLimit; ++k)
        if (mbar_test(bar, 0)) return true;
    return false;
}

// Four blocks per SM (at most 64 registers); kItems keys per thread (see
// sort_tile_items).  The tile's keys and values arrive in shared memory by two
// bulk copies (the copy engine moves them, up to 36 KB, while the block's
// threads are free), then each thread ranks its keys, and the tile leaves sorted by digit through the
// same shared buffers with coalesced stores.  The scatter itself cannot be a
// bulk copy: a digit's run starts at an arbitrary 8-byte offset of the output.
// Passes below the step's first pass (shift < 64 - 8 sort_passes) return at
// once; passes == nullptr runs every pass.
template <int kItems>
__global__ void __launch_bounds__(kSortThreads, 4)
onesweep_pass(const uint64_t* key_in, const uint32_t* val_in,
              uint64_t* key_out, uint32_t* val_out, int64_t n, int shift,
              const uint32_t* hist, uint32_t* status,
              unsigned* tile_counter, unsigned* err,
              const int32_t* passes, int tiles) {
    chain_begin();
    constexpr int kTile = kItems * kSortThreads;
    constexpr int kMatch = 256 * kWarps;  // the match words, in the values' place
    if (passes && shift < 64 - 8 * *passes) return;
    __shared__ uint16_t whist[kWarps][256];
    __shared__ uint32_t tile_start[256];
    __shared__ uint32_t goff[256];
    __shared__ uint32_t warp_tot[kWarps];
    __shared__ __align__(16) uint64_t skey[kTile];
    __shared__ __align__(16) uint32_t sval[kTile > kMatch ? kTile : kMatch];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int tile_sh;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        const int tile = (int)atomicAdd(tile_counter, 1u);
        tile_sh = tile;
        const int64_t base = (int64_t)tile * kTile;
        const int tile_n = (int)min((int64_t)kTile, n - base);
        const int bulk = tile_n & ~3;  // whole 16-byte chunks of both arrays
        mbar_init(&bar);
        mbar_expect_tx(&bar, (unsigned)bulk * 12u);
        if (bulk > 0) {
            bulk_load(skey, key_in + base, (unsigned)bulk * 8u, &bar);
            bulk_load(sval, val_in + base, (unsigned)bulk * 4u, &bar);
        }
    }
#pragma unroll
    for (int w = 0; w < kWarps; ++w) whist[w][tid] = 0;
    __syncthreads();
    const int tile = tile_sh;
    const int64_t base = (int64_t)tile * kTile;
    const int tile_n = (int)min((int64_t)kTile, n - base);
    {
        const int bulk = tile_n & ~3;
        if (tid < tile_n - bulk) {  // the last tile's ragged end, at most 3 keys
            skey[bulk + tid] = key_in[base + bulk + tid];
            sval[bulk + tid] = val_in[base + bulk + tid];
        }
        bool ok = mbar_wait_bounded(&bar);
        if (!ok) {
            atomicOr(err, kErrTimeout);
            ok = mbar_wait_bounded(&bar);  // let the copies land before the block moves on
        }
    }
    __syncthreads();
    const int seg = warp * (32 * kItems);
    uint64_t k_reg[kItems];
    uint32_t v_reg[kItems];
    uint32_t r_reg[kItems];
    const unsigned below = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int li = seg + k * 32 + lane;
        const bool valid = li < tile_n;
        k_reg[k] = valid ? skey[li] : 0ull;
        v_reg[k] = valid ? sval[li] : 0u;
    }
    __syncthreads();
    // the rows' match words take the values' place until the tile is scattered
    uint32_t* match = sval + warp * 256;
#pragma unroll
    for (int k = lane; k < 256; k += 32) match[k] = 0;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        r_reg[k] = row_rank(match, whist[warp], (uint32_t)(k_reg[k] >> shift) & 255u,
                            seg + k * 32 + lane < tile_n, below);
    __syncthreads();
    uint32_t count;
    {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = whist[w][tid];
            whist[w][tid] = (uint16_t)run;
            run += c;
        }
        count = run;
        tile_start[tid] = block_exclusive_scan(run, warp_tot, nullptr);
    }
    // Look-back for digit tid.  All tiles of a wave start together, so a tile
    // meets no finished prefix for hundreds of tiles back; walking these one by
    // one took 5 to 8 of a tile's 14 us at 1M.  So a tile adds its counts to its
    // group's words as well (with the number of tiles that have, above the
    // counts), and sums up the earlier tiles of its group and then the groups
    // before, until it meets one whose first tile has published its start.
    // Sort phase 62.1 -> 56.1 us at 300k, 116.8 -> 104.5 at 1M, 302 -> 289 at 4M
    // (groups of 16: 57.5, 104.5, 289; of 32: 62, 109, 291).
    const int group = tile / kSortGroup;
    const int groups = (tiles + kSortGroup - 1) / kSortGroup;
    uint32_t* sums = status + (int64_t)tiles * 256 + tid;
    uint32_t* starts = sums + (int64_t)groups * 256;
    st_status(status + (int64_t)tile * 256 + tid, kFlagAgg | count);
    atomicAdd(sums + (int64_t)group * 256, (1u << kGroupBits) + count);
    // first place of digit tid in the output
    const uint32_t bin = block_exclusive_scan(hist[tid], warp_tot, nullptr);
    // The tile goes into digit order in shared memory while the counts travel
    // (after the look-back: 60 us at 300k, 111 at 1M, 304 at 4M).  The scan's
    // barriers stand between tile_start's writes and these reads.
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int li = seg + k * 32 + lane;
        if (li < tile_n) {
            const uint32_t d = (uint32_t)((k_reg[k] >> shift) & 0xFF);
            const uint32_t lp = tile_start[d] + whist[warp][d] + r_reg[k];
            skey[lp] = k_reg[k];
            sval[lp] = v_reg[k];
        }
    }
    uint32_t excl = 0;
    for (int j = tile - 1; j >= group * kSortGroup; j -= kLook) {
        uint32_t v[kLook];
#pragma unroll
        for (int q = 0; q < kLook; ++q)
            v[q] = j - q >= group * kSortGroup ? ld_status(status + (int64_t)(j - q) * 256 + tid)
                                               : kFlagAgg;
#pragma unroll
        for (int q = 0; q < kLook; ++q) {
            for (int spins = 0; !(v[q] & kFlagAgg);) {
                if (++spins > kSpinLimit) {
                    atomicOr(err, kErrTimeout);
                    break;
                }
                v[q] = ld_status(status + (int64_t)(j - q) * 256 + tid);
            }
            excl += v[q] & ~kFlagAgg;
        }
    }
    bool found = false;
    for (int h = group - 1; h >= 0 && !found; h -= kLook) {
        uint32_t v[kLook], p[kLook];
#pragma unroll
        for (int q = 0; q < kLook; ++q) {
            v[q] = h - q >= 0 ? ld_status(sums + (int64_t)(h - q) * 256)
                              : (uint32_t)kSortGroup << kGroupBits;
            p[q] = h - q >= 0 ? ld_status(starts + (int64_t)(h - q) * 256) : kFlagAgg;
        }
#pragma unroll
        for (int q = 0; q < kLook; ++q) {
            if (found) continue;
            for (int spins = 0; (v[q] >> kGroupBits) != kSortGroup;) {
                if (++spins > kSpinLimit) {
                    atomicOr(err, kErrTimeout);
                    break;
                }
                v[q] = ld_status(sums + (int64_t)(h - q) * 256);
            }
            excl += v[q] & ((1u << kGroupBits) - 1);
            found = p[q] & kFlagAgg;
            if (found) excl += p[q] & ~kFlagAgg;
        }
    }
    if (tile % kSortGroup == 0) st_status(starts + (int64_t)group * 256, kFlagAgg | excl);
    goff[tid] = bin + excl;
    __syncthreads();
    for (int p = tid; p < tile_n; p += kSortThreads) {
        const uint64_t kk = skey[p];
        const uint32_t d = (uint32_t)((kk >> shift) & 0xFF);
        const uint32_t gp = goff[d] + (uint32_t)p - tile_start[d];
        key_out[gp] = kk;
        val_out[gp] = sval[p];
    }
}

// ---------------------------------------------------------------------------
// Tie pass.  After radix passes over the top P bytes only, keys that agree in
// those bytes sit together in their input order; putting each such group in
// order of its low bytes (ties kept in input order) gives exactly the full
// stable sort.  tie_mark lists the groups, tie_sort_small orders groups of
// up to 32 keys one warp each in registers, tie_sort_big orders larger ones
// one warp each by an LSD radix sort of the low bytes through the free
// ping-pong buffers.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
tie_mark(const uint64_t* key, int64_t n, DeviceScalars* s,
         uint2* small, uint2* big) {
    chain_begin();
    const int passes = s->sort_passes;
    if (passes >= 8) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int sh = 64 - 8 * passes;
    const int lane = threadIdx.x & 31;
    // each key is read once; the neighbours come from the next and previous
    // lanes (the row's end lanes read theirs)
    const uint64_t ki = i < n ? key[i] : 0ull;
    uint64_t kn = __shfl_down_sync(kFull, ki, 1), kp = __shfl_up_sync(kFull, ki, 1);
    if (lane == 31 && i + 1 < n) kn = key[i + 1];
    if (lane == 0 && i > 0 && i < n) kp = key[i - 1];
    bool start = false;
    int64_t e = i;
    if (i + 1 < n) {
        const uint64_t top = ki >> sh;
        start = (kn >> sh) == top && (i == 0 || (kp >> sh) != top);
        if (start) {  // last key of the group: galloping search
            int64_t step = 1, good = i + 1;
            while (good + step < n && (key[good + step] >> sh) == top) {
                good += step;
                step <<= 1;
            }
            int64_t lo = good, hi = min(n - 1, good + step - 1);
            while (lo < hi) {
                const int64_t mid = (lo + hi + 1) >> 1;
                if ((key[mid] >> sh) == top) lo = mid; else hi = mid - 1;
            }
            e = lo;
        }
    }
    const unsigned size = (unsigned)(e - i + 1);
    const bool is_small = start && size <= 32, is_big = start && size > 32;
    const unsigned ms = __ballot_sync(kFull, is_small), mb = __ballot_sync(kFull, is_big);
    unsigned b0 = 0, b1 = 0;
    if (lane == 0) {
        if (ms) b0 = atomicAdd(&s->tie_count[0], __popc(ms));
        if (mb) b1 = atomicAdd(&s->tie_count[1], __popc(mb));
    }
    b0 = __shfl_sync(kFull, b0, 0);
    b1 = __shfl_sync(kFull, b1, 0);
    const unsigned lt = lanemask_lt();
    if (is_small) small[b0 + __popc(ms & lt)] = make_uint2((unsigned)i, size);
    if (is_big) big[b1 + __popc(mb & lt)] = make_uint2((unsigned)i, size);
}

// Groups of 2..32 keys: lane l holds key l of the group and counts the keys
// that go before it (smaller, or equal and earlier).  The keys share their top
// bytes, so comparing whole keys compares the low bytes.
// Groups of more than 32 keys (rare: many bodies within 2^-4P of the box
// width of each other): one warp per group, a stable LSD radix sort of the
// 8 - P low bytes, 32 keys at a time, between the group's range of the
// sorted buffers and the same range of the free ping-pong buffers.
constexpr int kTieWarps = 4;

__global__ void __launch_bounds__(kTieWarps * 32)
tie_sort(uint64_t* key0, uint32_t* val0, uint64_t* key1,
         uint32_t* val1, const uint2* small, const uint2* big,
         const DeviceScalars* s) {
    chain_begin();
    const int passes = s->sort_passes;
    if (passes >= 8) return;
    __shared__ uint32_t off[kTieWarps][256];
    const unsigned nsmall = s->tie_count[0], nbig = s->tie_count[1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned warps = gridDim.x * kTieWarps, me = blockIdx.x * kTieWarps + w;
    for (unsigned g = me; g < nsmall; g += warps) {
        const uint2 grp = small[g];
        const bool on = lane < (int)grp.y;
        const uint64_t k = on ? key0[grp.x + lane] : ~0ull;
        const uint32_t v = on ? val0[grp.x + lane] : 0u;
        int rank = 0;
        for (int j = 0; j < (int)grp.y; ++j) {
            const uint64_t kj = __shfl_sync(kFull, k, j);
            rank += (kj < k || (kj == k && j < lane)) ? 1 : 0;
        }
        __syncwarp();
        if (on) {
            key0[grp.x + rank] = k;
            val0[grp.x + rank] = v;
        }
    }
    const unsigned below = lanemask_lt();
    for (unsigned g = me; g < nbig; g += warps) {
        const uint2 grp = big[g];
        const unsigned first = grp.x, size = grp.y;
        for (int d = 0; d < 8 - passes; ++d) {
            const int sh = 8 * d;
            const bool from0 = (d & 1) == 0;
            const uint64_t* ks = from0 ? key0 : key1;
            const uint32_t* vs = from0 ? val0 : val1;
            uint64_t* kd = from0 ? key1 : key0;
            uint32_t* vd = from0 ? val1 : val0;
            for (int b = lane; b < 256; b += 32) off[w][b] = 0;
            __syncwarp();
            for (unsigned b = 0; b < size; b += 32) {
                if (b + lane < size) atomicAdd(&off[w][(ks[first + b + lane] >> sh) & 0xFF], 1u);
            }
            __syncwarp();
            // exclusive scan of the 256 bins, 8 per lane
            uint32_t c[8], tot = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                c[q] = off[w][lane * 8 + q];
                tot += c[q];
            }
            uint32_t inc = tot;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFull, inc, o);
                if (lane >= o) inc += t;
            }
            uint32_t run = inc - tot;
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                off[w][lane * 8 + q] = run;
                run += c[q];
            }
            __syncwarp();
            for (unsigned b = 0; b < size; b += 32) {
                const bool on = b + lane < size;
                const uint64_t k = on ? ks[first + b + lane] : 0ull;
                const uint32_t v = on ? vs[first + b + lane] : 0u;
                const uint32_t dg = (uint32_t)((k >> sh) & 0xFF);
                const unsigned peers = digit_peers(dg, on);
                const int leader = __ffs(peers) - 1;
                uint32_t pos = 0;
                if (on && lane == leader) {
                    pos = off[w][dg];
                    off[w][dg] = pos + __popc(peers);
                }
                pos = __shfl_sync(kFull, pos, leader) + __popc(peers & below);
                if (on) {
                    kd[first + pos] = k;
                    vd[first + pos] = v;
                }
                __syncwarp();
            }
        }
        if ((8 - passes) & 1) {  // the result is in the second buffers: copy it back
            for (unsigned b = lane; b < size; b += 32) {
                key0[first + b] = key1[first + b];
                val0[first + b] = val1[first + b];
            }
        }
        __syncwarp();
    }
}

// CU:135-147: gather the bodies into Morton order.  In SPLIT mode it also
// writes the FP32 source record of each body relative to the box centre.
__global__ void gather_kernel(const uint32_t* order, int64_t n, BodyBuffers src,
                              BodyBuffers dst, float4* body4,
                              const DeviceScalars* s, Batch bt,
                              unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t j = order[i];
    const double2 p = src.pos[j], v = src.vel[j];
    const double m = src.mass[j];
    const int32_t o = src.orig[j];
    const double2 c = body4 ? frame_center(s, bt, (int)i) : make_double2(0.0, 0.0);
    dst.pos[i] = p;
    dst.vel[i] = v;
    dst.mass[i] = m;
    dst.orig[i] = o;
    if (body4) {
        body4[i] = make_float4((float)(p.x - c.x), (float)(p.y - c.y), (float)m,
                               __int_as_float((int)i));
    }
}

inline unsigned blocks_for(int64_t n, int threads) {
    return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

namespace {

// As few keys per thread as one cluster allows (a pass ranks them one after
// the other), then as few blocks as hold them.
inline int cluster_items(int64_t n) { return n <= (int64_t)kClusterMost * kClusterThreads ? 1 : 2; }
inline int cluster_blocks(int64_t n) {
    const int64_t tile = (int64_t)cluster_items(n) * kClusterThreads;
    int blocks = 1;
    while (blocks * tile < n) blocks *= 2;
    return blocks;
}

// cluster_sorts() has set the kernel's attributes.
template <int kSrc>
cudaError_t launch_cluster_sort(cudaStream_t st, bool chained, const double2* pos, int64_t n,
                                DeviceScalars* s, int adaptive, int new_step, int fixed_passes,
                                const uint64_t* key_in, uint64_t* key_out, uint32_t* val_out,
                                unsigned long long* mark0, unsigned long long* mark1) {
    const bool one = cluster_items(n) == 1;
    const int blocks = cluster_blocks(n);
    return chain_launch(st, chained, one ? cluster_sort<1, kSrc> : cluster_sort<2, kSrc>, blocks,
                        kClusterThreads, one ? sizeof(ClusterSmem<1>) : sizeof(ClusterSmem<2>), blocks,
                        pos, n, s, adaptive, new_step, fixed_passes, key_in, key_out, val_out, mark0,
                        mark1);
}

// Sets a kernel's attributes and asks whether one cluster of it fits the device.
template <int kItems, int kSrc>
bool cluster_fits(int blocks) {
    auto* kernel = cluster_sort<kItems, kSrc>;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)blocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = blocks;
    cfg.blockDim = kClusterThreads;
    cfg.dynamicSmemBytes = sizeof(ClusterSmem<kItems>);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cfg.dynamicSmemBytes) == cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess)
        return clusters > 0;
    cudaGetLastError();  // answered: the caller sorts by passes over global memory
    return false;
}

inline bool by_cluster(const nb_ctx* c) { return c->sort.hist == nullptr; }

}  // namespace

bool cluster_sorts(int64_t n, bool from_keys) {
    if (n > kClusterSortMax) return false;
    const bool one = cluster_items(n) == 1;
    auto* fits = from_keys ? (one ? cluster_fits<1, kSrcKeys> : cluster_fits<2, kSrcKeys>)
                           : (one ? cluster_fits<1, kSrcBodies> : cluster_fits<2, kSrcBodies>);
    return fits(cluster_blocks(n));
}

void launch_bbox(nb_ctx* c, const double2* pos, bool new_step) {
    if (c->batch.nuni > 0) {
        c->launches += 2;
        chain_launch(c->stream, false, bbox_batch_kernel, blocks_for(c->n, 256 * kBoxRows), 256, 0, 1, pos, c->n,
                     c->batch, mark_of(c, 0));
        chain_launch(c->stream, true, bbox_batch_finish, blocks_for(c->batch.nuni, 128), 128, 0, 1,
                     c->batch, c->scal, c->n, new_step);
        return;
    }
    c->launches += 1;
    if (by_cluster(c)) {  // the whole stage
        launch_cluster_sort<kSrcBodies>(c->stream, false, pos, c->n, c->scal, 1, new_step, 0, nullptr,
                                        c->sort.key[0], c->sort.val[0], mark_of(c, 0), mark_of(c, 1));
        return;
    }
    chain_launch(c->stream, false, bbox_kernel, c->bbox_blocks, kBoxThreads, 0, 1, pos, c->n,
                 c->bbox_partials, c->scal, 1, new_step, mark_of(c, 0));
}

void launch_morton(nb_ctx* c, const double2* pos) {
    if (by_cluster(c) && c->batch.nuni == 0) return;  // launch_bbox has made the codes
    c->launches += 1;
    SortState z;
    z.hist = c->sort.hist;
    z.tile_counter = c->sort.tile_counter;
    z.status = c->sort.status;
    z.tiles = c->sort.tiles;
    if (c->batch.nuni > 0) {
        chain_launch(c->stream, true, morton_batch_kernel, blocks_for(c->n, 256), 256, 0, 1, pos, c->n,
                     c->batch, c->scal, c->sort.key[0], c->sort.key[1], c->sort.val[0],
                     c->sort.val[1], z);
        return;
    }
    chain_launch(c->stream, true, morton_kernel, blocks_for(c->n, 256), 256, 0, 1, pos, c->n, c->scal,
                 c->sort.key[0], c->sort.key[1], c->sort.val[0], c->sort.val[1], z);
}

// One radix pass over two tiles of keys in which only the second tile runs:
// its look-back waits on a predecessor that never publishes, so the bounded
// wait must give up and raise kErrTimeout.  Returns the error bits.
unsigned sort_timeout_probe(cudaStream_t st) {
    constexpr int n = 2 * kSortItemsMax * kSortThreads;
    uint64_t *key_in = nullptr, *key_out = nullptr;
    uint32_t *val_in = nullptr, *val_out = nullptr, *hist = nullptr, *status = nullptr;
    unsigned *counter = nullptr, *err = nullptr;
    unsigned flags = ~0u;
    if (cudaMalloc(&key_in, n * sizeof(uint64_t)) == cudaSuccess &&
        cudaMalloc(&key_out, n * sizeof(uint64_t)) == cudaSuccess &&
        cudaMalloc(&val_in, n * sizeof(uint32_t)) == cudaSuccess &&
        cudaMalloc(&val_out, n * sizeof(uint32_t)) == cudaSuccess &&
        cudaMalloc(&hist, 256 * sizeof(uint32_t)) == cudaSuccess &&
        cudaMalloc(&status, sort_status_rows(2) * 256 * sizeof(uint32_t)) == cudaSuccess &&
        cudaMalloc(&counter, sizeof(unsigned)) == cudaSuccess &&
        cudaMalloc(&err, sizeof(unsigned)) == cudaSuccess) {
        // all keys zero: digit 0 holds every key, bins are all 0
        cudaMemsetAsync(key_in, 0, n * sizeof(uint64_t), st);
        cudaMemsetAsync(val_in, 0, n * sizeof(uint32_t), st);
        cudaMemsetAsync(hist, 0, 256 * sizeof(uint32_t), st);
        cudaMemsetAsync(status, 0, sort_status_rows(2) * 256 * sizeof(uint32_t), st);
        cudaMemsetAsync(err, 0, sizeof(unsigned), st);
        const unsigned one = 1u;  // the single block takes tile 1
        cudaMemcpyAsync(counter, &one, sizeof(unsigned), cudaMemcpyHostToDevice, st);
        onesweep_pass<kSortItemsMax><<<1, kSortThreads, 0, st>>>(key_in, val_in, key_out, val_out, n, 0, hist, status,
                                                  counter, err, nullptr, 2);
        cudaMemcpyAsync(&flags, err, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) flags = ~0u;
    }
    cudaFree(key_in);
    cudaFree(key_out);
    cudaFree(val_in);
    cudaFree(val_out);
    cudaFree(hist);
    cudaFree(status);
    cudaFree(counter);
    cudaFree(err);
    return flags;
}

// The sorted keys and permutation end in buffer 0.
void launch_sort(nb_ctx* c) {
    uint64_t* const* key = c->sort.key;
    uint32_t* const* val = c->sort.val;
    c->launches += 2;
    if (by_cluster(c)) {
        if (c->batch.nuni > 0) {  // (otherwise launch_bbox has done it)
            c->launches += 1;
            launch_cluster_sort<kSrcKeys>(c->stream, true, nullptr, c->n, c->scal, 1, 0, 0, key[0],
                                          key[0], val[0], mark_of(c, 1), nullptr);
        }
    } else {
        // the Morton pass has reset the histograms, tile counters and status words
        const int tiles = c->sort.tiles, items = sort_tile_items(c->n, c->sm_count);
        auto* pass_kernel = items == 4   ? onesweep_pass<4>
                            : items == 8 ? onesweep_pass<8>
                                         : onesweep_pass<kSortItemsMax>;
        c->launches += 1 + 8;
        chain_launch(c->stream, true, onesweep_histogram,
                     std::min<unsigned>(4 * c->sm_count, blocks_for(c->n, 32 * kHistRows * kWarps)),
                     kSortThreads, 0, 1, key[0], key[1], c->n, c->scal, c->sort.hist, mark_of(c, 1));
        for (int pass = 0; pass < 8; ++pass) {
            const int src = pass & 1, dst = src ^ 1;
            chain_launch(c->stream, true, pass_kernel, tiles, kSortThreads, 0, 1, key[src], val[src],
                         key[dst], val[dst], c->n, 8 * pass, c->sort.hist + 256 * pass,
                         c->sort.status + (size_t)pass * 256 * sort_status_rows(tiles),
                         c->sort.tile_counter + pass, &c->scal->error, &c->scal->sort_passes, tiles);
        }
    }
    // keys tied in the sorted top bytes, in order of their low bytes
    chain_launch(c->stream, true, tie_mark, blocks_for(c->n, 256), 256, 0, 1, key[0], c->n, c->scal,
                 c->sort.ties_small, c->sort.ties_big);
    chain_launch(c->stream, true, tie_sort, std::min<unsigned>(c->sm_count * 16, blocks_for(c->n, 256)),
                 kTieWarps * 32, 0, 1, key[0], val[0], key[1], val[1], c->sort.ties_small,
                 c->sort.ties_big, c->scal);
}

// All 8 passes, so no ties are left.
cudaError_t launch_morton_sort_raw(const double2* pos, int64_t n, uint64_t* const key[2],
                                   uint32_t* const val[2], uint64_t* key_out, uint32_t* val_out,
                                   uint16_t* counts, double* partials, int bbox_blocks,
                                   DeviceScalars* scal, cudaStream_t st) {
    if (cluster_sorts(n, false))
        return launch_cluster_sort<kSrcBodies>(st, false, pos, n, scal, 0, 0, 8, nullptr, key_out,
                                               val_out, nullptr, nullptr);
    const int tiles = (int)count_tiles(n);
    cudaError_t e = chain_launch(st, false, bbox_kernel, bbox_blocks, kBoxThreads, 0, 1, pos, n,
                                 partials, scal, 0, 0, nullptr);
    if (e == cudaSuccess)
        e = chain_launch(st, true, morton_kernel, blocks_for(n, 256), 256, 0, 1, pos, n, scal, key[0],
                         key[1], val[0], val[1], SortState());
    for (int pass = 0; pass < 8 && e == cudaSuccess; ++pass) {
        const int src = pass & 1, dst = src ^ 1;
        e = chain_launch(st, true, count_digits, tiles, kCountThreads, 0, 1, key[src], n, pass, counts);
        if (e == cudaSuccess)
            e = chain_launch(st, true, count_scatter, tiles, kCountThreads, 0, 1, key[src], val[src],
                             pass == 7 ? key_out : key[dst], pass == 7 ? val_out : val[dst], n, pass,
                             counts, tiles);
    }
    return e;
}

void launch_gather(nb_ctx* c, const BodyBuffers& src, const BodyBuffers& dst, float4* body4) {
    c->launches += 1;
    chain_launch(c->stream, true, gather_kernel, blocks_for(c->n, 256), 256, 0, 1, c->sort.val[0], c->n,
                 src, dst, body4, c->scal, c->batch, mark_of(c, 2));
}

}  // namespace nb
