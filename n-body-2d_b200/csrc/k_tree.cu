// k_tree.cu -- compressed quadtree from sorted Morton codes, and its moments.
//
// Replaces the reference's level-by-level build (BarnesHutCuda.cu:153-240 and
// the host loop at CU:713-777, up to 31 launches each followed by a
// device-to-host copy) and its per-level COM passes (CU:251-344, CU:787-807).
//
// Construction (Karras-style, no host round trips):
//   For the boundary i between sorted bodies i and i+1 let d_i be the number
//   of leading 2-bit digits their codes share.  Every boundary with d_i < 30
//   separates two children of the cell "bodies sharing d_i digits with body
//   i", whose level is d_i.  That cell is created once, by its first child
//   boundary.  Cells are numbered in the order of those boundaries, which lays
//   every subtree out as a contiguous id range: each tile of boundaries ranks
//   its own, the last tile to be done adds up the tiles.  A last pass links
//   children (<= 4 per cell) and parents.
//
// The reference tree is uncompressed: a cell with one non-empty child is
// followed by a chain of single-child cells down to the next split, all with
// the same mass and centre of mass.  The reference accepts a chain at its
// first level that passes width^2 < theta^2 d^2, and because widths shrink
// with depth that happens iff the deepest level of the chain passes.  This
// tree therefore keeps only the deepest level of every chain and stores that
// level, so opening decisions and force terms equal the reference's
// (cell widths come from the level, never from the body range).
#include <climits>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nb_internal.cuh"

namespace nb {
namespace {

constexpr int kThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kThreads * kScanItems;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int lcp_digits(uint64_t a, uint64_t b) {
    const uint64_t x = a ^ b;
    return x ? (__clzll((long long)x) >> 1) : 32;
}

__device__ __forceinline__ bool share(uint64_t a, uint64_t b, int digits) {
    return digits <= 0 ? true : (digits >= 32 ? a == b : ((a ^ b) >> (64 - 2 * digits)) == 0);
}

// Last index e in [i, hi] whose code shares `digits` leading digits with key[i].
__device__ int gallop_right(const uint64_t* __restrict__ key, int i, int hi, int digits) {
    const uint64_t ki = key[i];
    int j = i, step = 1;
    while (true) {
        const int cand = i + step;
        if (cand > hi || !share(key[cand], ki, digits)) break;
        j = cand;
        step <<= 1;
    }
    int a = j, b = min(hi, i + step - 1);
    while (a < b) {
        const int mid = (a + b + 1) >> 1;
        if (share(key[mid], ki, digits)) a = mid; else b = mid - 1;
    }
    return a;
}

// ---- cell structure from the boundary levels ---------------------------
// Boundary i lies between bodies i and i + 1; its level c_i is the number of
// leading digits codes i and i + 1 share (capped at kMaxLevel: codes sharing
// 30 or more digits sit in one leaf).  The cell whose children boundary i
// separates spans the bodies between the nearest boundaries on either side
// with a smaller level, and the boundaries of equal level between those are
// its other child separators.  So the whole build reduces to nearest smaller
// values over c (ANSV), which three passes find without a search:
//   tree_lcp         c_i per boundary, and per tile and level v the first
//                    and last boundary with a level below v;
//   tree_ansv_tiles  those tables scanned over the tiles (prefix maximum of
//                    the last, suffix minimum of the first);
//   tree_ansv        per boundary the nearest smaller (and smaller-or-equal)
//                    level on each side: inside its warp row from the row's
//                    ballot for that level, inside its tile from the rows'
//                    summaries, beyond the tile from the scanned tables.
// A tile is kAnsvTile boundaries; warp w holds rows 8w..8w+7 of 32.  Lane v
// of a row needs the row's mask "level < v": each lane writes its level as a
// thermometer word (bit v set for every v above its level) and a 32 x 32 bit
// transpose across the warp (five butterfly shuffles) hands lane v bit v of
// every lane, which is that mask.
constexpr int kAnsvItems = kAnsvTile / kThreads;  // rows per warp (256 threads per tile)
constexpr int kAnsvRows = kAnsvTile / 32;           // 64 rows
constexpr int kNoLevel = kMaxLevel + 1;             // past the last body: never below a level
static_assert(kAnsvItems == 8 && kAnsvLevels == 32, "one lane per level, 8 rows per warp");

// Bit v set for every v above level c (v = 0..31).
__device__ __forceinline__ unsigned thermometer(int c) {
    return c >= 31 ? 0u : (0xFFFFFFFFu << (c + 1));
}

// Per level v and tile t the first and last boundary with a level below v.
// Level-major for the scan over the tiles; tile-major when tree_ansv reads the
// other tiles' entries itself.
struct TileTable {
    int32_t *first, *last;
    int level_stride, tile_stride;
    __device__ __forceinline__ int at(int v, int t) const { return v * level_stride + t * tile_stride; }
};
// Up to this many tiles, tree_ansv goes through the other tiles' entries (a few
// loads per thread) instead of a scan kernel before it.
constexpr int kFewTiles = 64;

// kBlock threads per tile: 1,024 while every SM has at most one tile (a warp's
// rows follow one another), else 256.
constexpr int kWideThreads = 1024;

template <int kBlock>
__global__ void __launch_bounds__(kBlock)
tree_lcp(const uint64_t* key, int n, uint8_t* lcp8,
         TileTable tab, unsigned* lcp_hist,
         unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    constexpr int kItems = kAnsvTile / kBlock;
    __shared__ unsigned hist[33];
    __shared__ int sfirst[kAnsvLevels], slast[kAnsvLevels];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 33) hist[threadIdx.x] = 0;
    if (threadIdx.x < kAnsvLevels) {
        sfirst[threadIdx.x] = INT_MAX;
        slast[threadIdx.x] = -1;
    }
    __syncthreads();
    const int base = blockIdx.x * kAnsvTile + warp * (32 * kItems);
    // lane v (1..30): first and last boundary of the warp's rows with level < v;
    // lane v (1..31) and lane 0 (for 32): how many have a level < v
    int myfirst = INT_MAX, mylast = -1;
    unsigned mycnt = 0, nbound = 0;
#pragma unroll 1
    for (int r = 0; r < kItems; ++r) {
        const int row0 = base + 32 * r;
        const int i = row0 + lane;
        int c = 64;  // not a boundary
        if (i < n - 1) c = lcp_digits(key[i], key[i + 1]);
        if (i < n) lcp8[i] = (uint8_t)(i < n - 1 ? min(c, kMaxLevel) : kNoLevel);
        // lane v (1..31): the row's mask of levels below v; lane 0: below 32
        unsigned mine = warp_transpose_bits(thermometer(c));
        const unsigned below32 = __ballot_sync(kFull, c < 32);
        if (lane == 0) mine = below32;
        nbound += __popc(__ballot_sync(kFull, i < n - 1));
        mycnt += __popc(mine);
        if (mine && lane >= 1 && lane <= kMaxLevel) {
            if (myfirst == INT_MAX) myfirst = row0 + __ffs(mine) - 1;
            mylast = row0 + 31 - __clz(mine);
        }
    }
    if (myfirst != INT_MAX) atomicMin(&sfirst[lane], myfirst);
    if (mylast >= 0) atomicMax(&slast[lane], mylast);
    {   // histogram of levels 0..32 from the counts below each level
        const unsigned c32 = __shfl_sync(kFull, mycnt, 0);
        const unsigned x = lane == 0 ? 0u : mycnt;         // count below level `lane`
        const unsigned up = __shfl_down_sync(kFull, x, 1);  // count below level lane + 1
        const unsigned h = lane < 31 ? up - x : c32 - x;
        if (h) atomicAdd(&hist[lane], h);
        if (lane == 0 && nbound > c32) atomicAdd(&hist[32], nbound - c32);
    }
    __syncthreads();
    if (threadIdx.x < kAnsvLevels) {
        tab.first[tab.at(threadIdx.x, blockIdx.x)] = sfirst[threadIdx.x];
        tab.last[tab.at(threadIdx.x, blockIdx.x)] = slast[threadIdx.x];
    }
    // the next step's sort reads how many neighbouring codes share d digits
    if (threadIdx.x < 33 && hist[threadIdx.x]) atomicAdd(lcp_hist + threadIdx.x, hist[threadIdx.x]);
}

// One block per level v: tile_last becomes the last boundary of tiles 0..t
// with a level below v, tile_first the first of tiles t..tiles-1.
constexpr int kTileScanThreads = 1024;
__global__ void __launch_bounds__(kTileScanThreads)
tree_ansv_tiles(int tiles, int32_t* tile_first, int32_t* tile_last) {
    chain_begin();
    __shared__ int wagg[kTileScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t* last = tile_last + blockIdx.x * tiles;
    int32_t* first = tile_first + blockIdx.x * tiles;
    int carry = -1;
    for (int b = 0; b < tiles; b += kTileScanThreads) {
        const int t = b + threadIdx.x;
        int x = t < tiles ? last[t] : -1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x = max(x, y);
        }
        if (lane == 31) wagg[warp] = x;
        __syncthreads();
        int pre = carry, tot = carry;
        for (int w = 0; w < kTileScanThreads / 32; ++w) {
            if (w < warp) pre = max(pre, wagg[w]);
            tot = max(tot, wagg[w]);
        }
        if (t < tiles) last[t] = max(x, pre);
        carry = tot;
        __syncthreads();
    }
    carry = INT_MAX;
    for (int b = tiles - 1; b >= 0; b -= kTileScanThreads) {
        const int t = b - (int)threadIdx.x;  // descending: a prefix over the threads is a suffix over tiles
        int x = t >= 0 ? first[t] : INT_MAX;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x = min(x, y);
        }
        if (lane == 31) wagg[warp] = x;
        __syncthreads();
        int pre = carry, tot = carry;
        for (int w = 0; w < kTileScanThreads / 32; ++w) {
            if (w < warp) pre = min(pre, wagg[w]);
            tot = min(tot, wagg[w]);
        }
        if (t >= 0) first[t] = min(x, pre);
        carry = tot;
        __syncthreads();
    }
}

// ---- numbering the cells ---------------------------------------------------
__device__ __forceinline__ int warp_inclusive(int v) {
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

template <int kBlock = kThreads>
__device__ int block_exclusive(int v, int* wsum, int* total) {
    static_assert(kBlock % 32 == 0 && kBlock <= 1024, "one warp scans the warp sums");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inc = warp_inclusive(v);
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < kBlock / 32 ? wsum[lane] : 0;
        const int winc = warp_inclusive(w);
        if (lane < kBlock / 32) wsum[lane] = winc - w;
        if (lane == kBlock / 32 - 1 && total) *total = winc;
    }
    __syncthreads();
    const int r = wsum[warp] + inc - v;
    __syncthreads();
    return r;
}

// Whether this block is the grid's last to come here; the writes of all blocks
// before are then visible to it.  The ticket is left at zero.
__device__ bool last_block(unsigned* ticket, unsigned blocks) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == blocks - 1;
        if (last) {
            __threadfence();
            *ticket = 0;
        }
    }
    __syncthreads();
    return last;
}

// One block: out[k] = sum of in[0..k), returns the total.
template <int kBlock>
__device__ int scan_tiles(const int32_t* in, int count, int32_t* out) {
    __shared__ int wsum[kBlock / 32];
    __shared__ int total;
    const int per = (count + kBlock - 1) / kBlock;
    const int k0 = min(count, (int)threadIdx.x * per), k1 = min(count, k0 + per);
    int sum = 0;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) sum += __ldcg(in + k);
    int run = block_exclusive<kBlock>(sum, wsum, &total);
    for (int k = k0; k < k1; ++k) {
        const int v = __ldcg(in + k);
        out[k] = run;
        run += v;
    }
    return total;
}

// Cells are numbered by their first separators: the cells of the tiles before,
// then the rank in the tile.
__device__ __forceinline__ int cell_id(const Tree& t, int boundary) {
    return t.tile_cells[boundary / kAnsvTile] + t.cell_rank[boundary];
}

// A boundary i below kMaxLevel creates a cell iff it is the cell's first
// separator (no equal level between it and the cell's start), which numbers
// the cells: cell_rank[i] = such boundaries before i in its tile, rep[] lists a
// tile's, and the grid's last block adds up the tiles (three scan kernels and a
// number per boundary before: tree and groups 254 -> 209 us at 4M, 51 -> 38 at
// 300,007 bodies, 36 -> 22 at 16,384).  bnd[i] = {first body of the cell, last body of the cell,
// previous separator of the cell or -1, next separator or -1}, the first two
// written for flagged boundaries only.  The cell's first body follows the
// nearest smaller level on the left, its last body is the nearest smaller on
// the right (or n - 1); a separator's neighbours are the nearest levels <= c_i
// when those equal c_i.
template <int kBlock>
__global__ void __launch_bounds__(kBlock)
tree_ansv(Tree t, int n, int tiles, TileTable tab, DeviceScalars* s) {
    chain_begin();
    constexpr int kItems = kAnsvTile / kBlock, kWarps = kBlock / 32;
    // masks[r][v]: row r's ballot of "level < v" (v = 1..30; 0 elsewhere).
    // rlast[r][v]: after the scan, the last boundary with a level below v in
    // rows of r's part p up to r (-1 if none), rfirst[r][v] the first in rows
    // from r on (kAnsvTile if none); tile-local positions
    __shared__ unsigned masks[kAnsvRows][32];
    __shared__ int16_t rlast[kAnsvRows][kAnsvLevels];
    __shared__ int16_t rfirst[kAnsvRows][kAnsvLevels];
    __shared__ int16_t before[kWarps][kAnsvLevels];  // last in the parts before p
    __shared__ int16_t after[kWarps][kAnsvLevels];   // first in the parts after p
    __shared__ unsigned creates[kAnsvRows];  // the row's first separators
    __shared__ int far_last[kWarps][32], far_first[kWarps][32];
    const uint8_t* __restrict__ lcp8 = t.lcp8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x, tbase = tile * kAnsvTile;
    // few tiles: the last boundary below level `lane` in the tiles before, the
    // first in the tiles after, over a part of the tiles per warp
    const bool few = tiles <= kFewTiles;
    if (few) {
        int l = -1, f = INT_MAX;
#pragma unroll 4
        for (int q = warp; q < tiles; q += kWarps) {
            if (q < tile) l = max(l, tab.last[tab.at(lane, q)]);
            if (q > tile) f = min(f, tab.first[tab.at(lane, q)]);
        }
        far_last[warp][lane] = l;
        far_first[warp][lane] = f;
    }
#pragma unroll 1
    for (int r = 0; r < kItems; ++r) {
        const int row = warp * kItems + r;
        const int i = tbase + 32 * row + lane;
        const int cap = i < n ? lcp8[i] : kNoLevel;
        // lane v: the row's mask of levels below v (lanes 0 and 31 unused: 0)
        unsigned mine = warp_transpose_bits(thermometer(cap));
        if (lane == 0 || lane > kMaxLevel) mine = 0u;
        masks[row][lane] = mine;
        rfirst[row][lane] = (int16_t)(mine ? 32 * row + __ffs(mine) - 1 : kAnsvTile);
        rlast[row][lane] = (int16_t)(mine ? 32 * row + 31 - __clz(mine) : -1);
    }
    __syncwarp();
    {   // scan the warp's own 8 rows, lane = level
        int run = -1;
        for (int r = 0; r < kItems; ++r) {
            const int row = warp * kItems + r;
            run = max(run, (int)rlast[row][lane]);
            rlast[row][lane] = (int16_t)run;
        }
        int runf = kAnsvTile;
        for (int r = kItems - 1; r >= 0; --r) {
            const int row = warp * kItems + r;
            runf = min(runf, (int)rfirst[row][lane]);
            rfirst[row][lane] = (int16_t)runf;
        }
    }
    __syncthreads();
    {
        int b = -1, a = kAnsvTile;
        for (int p = 0; p < kWarps; ++p) {
            if (p < warp) b = max(b, (int)rlast[p * kItems + kItems - 1][lane]);
            if (p > warp) a = min(a, (int)rfirst[p * kItems][lane]);
        }
        before[warp][lane] = (int16_t)b;
        after[warp][lane] = (int16_t)a;
    }
    if (few && warp == 0) {
        int l = -1, f = INT_MAX;
        for (int p = 0; p < kWarps; ++p) {
            l = max(l, far_last[p][lane]);
            f = min(f, far_first[p][lane]);
        }
        far_last[0][lane] = l;
        far_first[0][lane] = f;
    }
    __syncthreads();
    const unsigned lt = lanemask_lt(), gt = ~lt & ~(1u << lane);
#pragma unroll 1
    for (int r = 0; r < kItems; ++r) {
        const int row = warp * kItems + r;
        const int i = tbase + 32 * row + lane;
        const int v = i < n - 1 ? lcp8[i] : kNoLevel;
        bool first_sep = false;
        if (v < kMaxLevel) {
            // nearest boundary on the left / right with a level below u
            auto left = [&](int u) {
                const unsigned m = masks[row][u] & lt;
                if (m) return tbase + 32 * row + 31 - __clz(m);
                int j = r > 0 ? (int)rlast[row - 1][u] : -1;
                if (j < 0) j = before[warp][u];
                if (j >= 0) return tbase + j;
                if (few) return far_last[0][u];
                return tile > 0 ? tab.last[tab.at(u, tile - 1)] : -1;
            };
            auto right = [&](int u) {
                const unsigned m = masks[row][u] & gt;
                if (m) return tbase + 32 * row + __ffs(m) - 1;
                int j = r < kItems - 1 ? (int)rfirst[row + 1][u] : kAnsvTile;
                if (j >= kAnsvTile) j = after[warp][u];
                if (j < kAnsvTile) return tbase + j;
                const int g = few                ? far_first[0][u]
                              : tile + 1 < tiles ? tab.first[tab.at(u, tile + 1)]
                                                 : INT_MAX;
                return g == INT_MAX ? n - 1 : g;
            };
            const int l_lt = left(v), l_le = left(v + 1);
            const int r_lt = right(v), r_le = right(v + 1);
            first_sep = l_le == l_lt;
            t.bnd[i] = make_int4(first_sep ? l_lt + 1 : -1, first_sep ? r_lt : -1,
                                 first_sep ? -1 : l_le, r_le == r_lt ? -1 : r_le);
        }
        const unsigned c = __ballot_sync(kFull, first_sep);
        if (lane == 0) creates[row] = c;
    }
    __syncthreads();
    int run = 0;  // of the warps before
    for (int q = lane; q < warp * kItems; q += 32) run += __popc(creates[q]);
    run = __reduce_add_sync(kFull, run);
    for (int r = 0; r < kItems; ++r) {
        const int row = warp * kItems + r;
        const int i = tbase + 32 * row + lane;
        const unsigned c = creates[row];
        const int rank = run + __popc(c & lt);
        if (i < n) t.cell_rank[i] = (uint16_t)rank;
        if ((c >> lane) & 1u) t.rep[tbase + rank] = (uint16_t)(i - tbase);
        run += __popc(c);
    }
    if (threadIdx.x == kBlock - 1) t.tile_count[tile] = run;
    if (threadIdx.x == 0 && t.tile_groups) t.tile_groups[tile] = 0;  // the linking pass counts
    if (last_block(&s->tile_ticket, gridDim.x)) {
        const int total = scan_tiles<kBlock>(t.tile_count, tiles, t.tile_cells);
        if (threadIdx.x == 0) s->cells = total;
    }
}

// Moments of a multi-body leaf in the reference's summation order: 128
// strided partial sums, then a halving tree (CU:284-309).  The halving tree
// adds the partials as a balanced binary tree whose leaves, left to right, are
// the partials in 7-bit bit-reversed order, so a binary-counter pairwise sum
// over that sequence reproduces it with an 8-entry stack.  Such leaves only
// hold bodies whose codes agree in 60 bits, so they are rare and small.
__device__ void bucket_moments(const double2* __restrict__ pos, const double* __restrict__ mass,
                               int first, int last, double* out_m, double2* out_c) {
    double sm[8], sx[8], sy[8];
    for (int k = 0; k < 128; ++k) {
        const int tx = (int)(__brev((unsigned)k) >> 25);
        double M = 0.0, Rx = 0.0, Ry = 0.0;
        for (int i = first + tx; i <= last; i += 128) {
            const double m = mass[i];
            M += m;
            Rx = fma(m, pos[i].x, Rx);
            Ry = fma(m, pos[i].y, Ry);
        }
        int lvl = 0;
        while ((k >> lvl) & 1) {
            M = sm[lvl] + M;
            Rx = sx[lvl] + Rx;
            Ry = sy[lvl] + Ry;
            ++lvl;
        }
        sm[lvl] = M;
        sx[lvl] = Rx;
        sy[lvl] = Ry;
    }
    *out_m = sm[7];
    *out_c = make_double2(sx[7] / sm[7], sy[7] / sm[7]);
}

// Every cell (one thread each) writes its own record and its leaf children,
// and enters itself in its parent's child list: the parent is the cell of the
// deeper of the two boundaries around this cell's bodies (their levels are
// below the cell's; ties are two separators of the same parent), and the
// slot is the child's position among the parent's children in code order.
// Mass, COM and the packed FP32 record of cell id from two prefix sums
// (SPLIT monopoles; defined with the prefix kernels below, which run before
// the tree build).
__device__ void cell_from_prefix(const double4* __restrict__ prefix, const Tree& t,
                                 const DeviceScalars* __restrict__ s, const Batch& bt,
                                 const double2* __restrict__ pos, int id, int2 r, int level,
                                 float accept_scale);

// Groups of half the size or less, whose bodies lie one to a lane, are listed
// after all others up to kSmallLastMax bodies (small > 0): the walk takes the
// groups in order, and ends sooner when the cheap ones come last.  Above, the
// end matters less than the places in the tree that neighbours share.  Force
// phase, us, in key order and small ones last: collision 262,144 bodies 130 and
// 126, 524,288 223 and 204, 1M 404 and 386, 2M 777 and 767, 4M 1,541 and 1,546,
// 1M with quadrupoles 865 and 841, Plummer 300,000 171 and 161; listing them costs
// 1.2 us.  Groups of up to 32 bodies cost alike, and learned contexts sample groups
// by index: both keep the order of the keys.
constexpr int64_t kSmallLastMax = 2097152;
// Counts of groups: all above kSmallBits and small ones (at most 9 a cell) below,
// where small ones are listed apart; else all.
constexpr int kSmallBits = 15;
static_assert(9 * kAnsvTile < 1 << kSmallBits &&
                  kSmallLastMax / 64 + 9 * kAnsvTile < 1 << (31 - kSmallBits),
              "a tile's counts fit a word");

// The SPLIT target groups of one cell (defined with tree_groups_write below).
template <bool kWrite>
__device__ __forceinline__ int cell_groups(int2 rg, bool is_root, int nc, const int* ca, const int* cb,
                           const bool* leaf, int gsize, int fill, int small, const Batch& bt,
                           const uint64_t* __restrict__ key, int2* __restrict__ out,
                           int2* __restrict__ out_small);

// A tree without internal cells: one body, or all bodies in one level-30 leaf.
__device__ void trivial_root(const double2* __restrict__ pos, const double* __restrict__ mass, int n,
                             const Tree& t, DeviceScalars* __restrict__ s) {
    s->root = ~0;
    t.leaf_last[0] = n - 1;
    t.leaf_plevel[0] = -1;
    if (n > 1) bucket_moments(pos, mass, 0, n - 1, t.bucket_mass, t.bucket_com);
}

// Cell id, created by boundary i; returns its target groups (gsize > 0).
template <bool kMono>
__device__ __forceinline__ int link_cell(int i, int id, const uint64_t* __restrict__ key, int n,
                                         const double2* __restrict__ pos,
                                         const double* __restrict__ mass, const Tree& t,
                                         DeviceScalars* __restrict__ s,
                                         const double4* __restrict__ prefix, const Batch& bt,
                                         float accept_scale, int gsize, int fill, int small) {
    const uint8_t* __restrict__ lcp8 = t.lcp8;
    const int4 bi = t.bnd[i];
    const int c = lcp8[i];
    const int first = bi.x, last = bi.y;
    // the cell's separators: i, then the chain of next separators
    int sep[3] = {i, n - 1, n - 1};
    int ns = 1;
    int next = bi.w;
#pragma unroll
    for (int q = 1; q < 3; ++q)
        if (next >= 0) {
            sep[q] = next;
            ++ns;
            next = t.bnd[next].w;
        }
    if (next >= 0) atomicOr(&s->error, kErrTree);  // a fifth child: inconsistent codes
    int* child = reinterpret_cast<int*>(t.child + id);
    int nint = 0;
    int ca[4], cb[4];
    bool leaf[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q > ns) continue;
        const int a = q == 0 ? first : sep[q - 1] + 1;
        const int b = q == ns ? last : sep[min(q, 2)];
        ca[q] = a;
        cb[q] = b;
        leaf[q] = true;
        if (a == b) {
            child[q] = ~a;
            t.leaf_last[a] = a;
            t.leaf_plevel[a] = c;
        } else if (lcp8[a] == kMaxLevel && lcp_digits(key[a], key[b]) >= kMaxLevel) {
            // (a boundary below level 30 right after a makes the child a cell)
            child[q] = ~a;
            t.leaf_last[a] = b;
            t.leaf_plevel[a] = c;
            bucket_moments(pos, mass, a, b, t.bucket_mass + a, t.bucket_com + a);
        } else {
            leaf[q] = false;
            ++nint;  // a cell: it enters itself below
        }
    }
    int groups = 0;
    if (gsize > 0) {
        groups = cell_groups<false>(make_int2(first, last), first == 0 && last == n - 1,
                                    ns + 1, ca, cb, leaf, gsize, fill, small, bt, key, nullptr,
                                    nullptr);
        t.gcount[id] = groups;
    }
    for (int q = ns + 1; q < 4; ++q) child[q] = INT_MIN;
    t.range[id] = make_int2(first, last);
    t.level[id] = c;
    t.nint[id] = nint;
    t.ready[id] = 0;
    if (kMono) cell_from_prefix(prefix, t, s, bt, pos, id, make_int2(first, last), c, accept_scale);
    if (first == 0 && last == n - 1) {
        s->root = id;
        t.parent[id] = -1;
        return groups;
    }
    const int cl = first > 0 ? lcp8[first - 1] : -1;
    const int cr = last < n - 1 ? lcp8[last] : -1;
    const bool from_left = cl >= cr;
    int k = from_left ? first - 1 : last;  // a separator of the parent
    int rank = 0;  // its rank among the parent's separators; k ends at the first
    for (int p = t.bnd[k].z; p >= 0 && rank < 3; p = t.bnd[k].z) {
        k = p;
        ++rank;
    }
    const int slot = from_left ? rank + 1 : rank;
    if (slot > 3) {  // more than four children: the codes are inconsistent
        atomicOr(&s->error, kErrTree);
        return groups;
    }
    const int pid = cell_id(t, k);
    reinterpret_cast<int*>(t.child + pid)[slot] = id;
    t.parent[id] = pid;
    return groups;
}

// Five blocks per SM (48 registers): more dependent load chains in flight
// than the 56-register build's four (tree phase 0.196 -> 0.192 ms at 4M).
// kMono (SPLIT monopoles): the prefix sums are ready, and each cell also
// writes its monopole record, which saves a pass over the cells.  gsize > 0
// (SPLIT): each cell also counts its target groups into gcount.
constexpr int kLinkBlocks = kAnsvTile / kThreads;

template <bool kMono>
__global__ void __launch_bounds__(kThreads, 5)
tree_link(const uint64_t* key, int n, const double2* pos,
          const double* mass, Tree t, DeviceScalars* s,
          const double4* prefix, Batch bt, float accept_scale, int gsize, int fill,
          int small) {
    chain_begin();
    const int tile = blockIdx.x / kLinkBlocks;
    const int cells = s->cells;
    if (cells == 0) {  // one body, or all bodies in one level-30 leaf
        if (blockIdx.x == 0 && threadIdx.x == 0) trivial_root(pos, mass, n, t, s);
        return;
    }
    // the tile's cell j; kLinkBlocks blocks share a tile
    const int j = (blockIdx.x % kLinkBlocks) * kThreads + threadIdx.x;
    int groups = 0;
    if (j < t.tile_count[tile])
        groups = link_cell<kMono>(tile * kAnsvTile + t.rep[tile * kAnsvTile + j],
                                  t.tile_cells[tile] + j, key, n, pos, mass, t, s, prefix, bt,
                                  accept_scale, gsize, fill, small);
    if (gsize == 0) return;
    const int sum = __reduce_add_sync(kFull, groups);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(t.tile_groups + tile, sum);
}

// b_max^2 of a cell: squared distance from its COM to the farthest corner of
// its square.  The square is the cell's Morton prefix decoded in the box the
// codes were made in (the single box, or the cell's universe); forest cells
// above the universe roots are never accepted and get 0.
__device__ __forceinline__ double cell_bmax2(const DeviceScalars* s, const Batch& bt,
                                             const double2* __restrict__ pos, int first, int level,
                                             double2 com) {
    double2 lo;
    double w, scale;
    int bits, lvl = level;
    if (bt.nuni == 0) {
        lo = make_double2(s->box[0], s->box[2]);
        w = s->box[1] - s->box[0];
        scale = 4294967296.0;
        bits = 32;
    } else {
        if (level < kBatchUidDigits) return 0.0;
        const int u = bt.uid[first];
        lo = bt.lo[u];
        w = sqrt(bt.w2[u]);
        scale = (double)(1u << kBatchMortonBits);
        bits = kBatchMortonBits;
        lvl = level - kBatchUidDigits;
    }
    if (!(w > 0.0)) return 0.0;
    // the cell's column and row: the first body's grid coordinate, as the
    // Morton kernels compute it, cut to the cell's level
    const double inv_w = 1.0 / w, top = scale - 1.0;
    const double2 p = pos[first];
    const unsigned ix = __double2uint_rd(fmin(fmax((p.x - lo.x) * inv_w * scale, 0.0), top));
    const unsigned iy = __double2uint_rd(fmin(fmax((p.y - lo.y) * inv_w * scale, 0.0), top));
    const double wc = ldexp(w, -lvl);
    const double kx = lvl == 0 ? 0.0 : (double)(ix >> (bits - lvl));
    const double ky = lvl == 0 ? 0.0 : (double)(iy >> (bits - lvl));
    const double ax = fma(kx, wc, lo.x), ay = fma(ky, wc, lo.y);
    const double dx = fmax(fabs(ax - com.x), fabs(ax + wc - com.x));
    const double dy = fmax(fabs(ay - com.y), fabs(ay + wc - com.y));
    return dx * dx + dy * dy;
}

// The acceptance size the walk compares with theta^2 d^2: w^2, or with the
// b_max test max(w^2, b_max^2 theta^2 / ratio^2) (accept_scale =
// theta^2 / ratio^2), so that one comparison applies both tests.
__device__ __forceinline__ float accept_size2(const DeviceScalars* s, const Batch& bt,
                                              const double2* __restrict__ pos, int first,
                                              int level, double2 com, float accept_scale) {
    const double w2 = cell_width2(s, bt, first, level);
    if (accept_scale <= 0.f) return (float)w2;
    return (float)fmax(w2, cell_bmax2(s, bt, pos, first, level, com) * (double)accept_scale);
}

// Two floats rounded to BF16 (round to nearest even), lo in the low half.
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Mass, COM and (kSecond) second moments of a cell.
struct Moments {
    double m, x, y, sxx, sxy, syy;
};

// Moments of one cell from its children's masses and COMs c, in quadrant order
// with the reference's arithmetic (CU:329-343): M += m; R = fma(m, com, R);
// com = R / M (a missing child has mass 0 and changes nothing).  kSecond (the
// quadrupole walk) also accumulates second moments about the COM by the
// parallel-axis rule, S = sum_c [S_c + m_c d_c d_c^T] with d_c = com_c - com, in
// FP64; second(q) is child q's {Sxx, Sxy, Syy}.  Leaves have S = 0 (a
// multi-body leaf spans less than width / 2^30, so its own S is negligible).
template <bool kSecond, typename Second>
__device__ __forceinline__ Moments combine_children(const double3 (&c)[4], Second second) {
    double M = c[0].x, Rx = c[0].x * c[0].y, Ry = c[0].x * c[0].z;
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        M += c[q].x;
        Rx = fma(c[q].x, c[q].y, Rx);
        Ry = fma(c[q].x, c[q].z, Ry);
    }
    Moments o{M, Rx / M, Ry / M, 0.0, 0.0, 0.0};
    if (kSecond) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double3 v = second(q);
            o.sxx += v.x;
            o.sxy += v.y;
            o.syy += v.z;
            const double dx = c[q].y - o.x, dy = c[q].z - o.y;
            o.sxx += c[q].x * dx * dx;
            o.sxy += c[q].x * dx * dy;
            o.syy += c[q].x * dy * dy;
        }
    }
    return o;
}

__device__ __forceinline__ double3 bucket_leaf(const Tree& t, int b) {
    const double2 p = t.bucket_com[b];
    return make_double3(t.bucket_mass[b], p.x, p.y);
}

// A cell's moments as its parent and the walks read them; the second moments
// themselves only where a parent will read them from memory (`up`).
template <bool kSplit, bool kSecond>
__device__ __forceinline__ void store_moments(int id, const Moments& o, bool up,
                                              const DeviceScalars* __restrict__ s,
                                              const double2* __restrict__ pos, const Tree& t,
                                              const Batch& bt, float accept_scale) {
    const double2 com = make_double2(o.x, o.y);
    __stcg(t.mass + id, o.m);
    __stcg(t.com + id, com);
    if (kSecond && up) {
        double2* so = reinterpret_cast<double2*>(t.s64 + id);
        __stcg(so, make_double2(o.sxx, o.sxy));
        __stcg(so + 1, make_double2(o.syy, 0.0));
    }
    if (kSplit) {
        const int first = t.range[id].x;
        const double2 fc = frame_center(s, bt, first);
        t.cell4[id] = make_float4((float)(com.x - fc.x), (float)(com.y - fc.y), (float)o.m,
                                  accept_size2(s, bt, pos, first, t.level[id], com, accept_scale));
        // the walk's record carries 7.5 S, the factor of its (d.S.d) r^-7 term
        if (kSecond)
            t.cellq[id] =
                make_float4((float)(7.5 * o.sxx), (float)(7.5 * o.sxy), (float)(7.5 * o.syy), 0.f);
    }
}

// Arrival at a parent: release publishes this cell's moments, acquire makes
// the siblings' moments visible to the thread that goes on to the parent.
__device__ __forceinline__ int arrive_acq_rel(int* counter) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;"
                 : "=r"(old)
                 : "l"(counter)
                 : "memory");
    return old;
}

// Bottom-up pass, one block per kMomentBodies bodies.  Cells are numbered in
// body order, so the cells whose first separator lies in the block's bodies
// are one range of ids, and those whose bodies all do (some 99%) form whole
// subtrees, which the block computes in shared memory.  Cells that reach beyond
// the block are left to a climb over global memory: the last child to arrive
// at a parent goes on with it, some 2 us a step, where a publication and three
// dependent loads follow one another.  With that climb for all cells the pass
// took 37 us at 1,001 bodies, 51 at 16,384, 99 at 1,048,576 (quadrupoles 173);
// now 14, 27, 66 and 130.  A round is a chain of FP64 latencies (0.5 us), so
// larger blocks of bodies gain while the rounds grow with the depth only (512
// bodies: 22, 26, 78 and 151 us).
constexpr int kMomentBodies = 1024;
constexpr int kMomentThreads = 256;
constexpr int kOutside = -1;

// Node j of a block: its cell j, or with kMomentBodies more the leaf that starts
// at its body j; the last node is the missing child.
constexpr int kMomentNodes = 2 * kMomentBodies + 1;

template <bool kSecond>
struct MomentSmem {
    double m[kMomentNodes], x[kMomentNodes], y[kMomentNodes];
    double s[kSecond ? 3 : 1][kSecond ? kMomentBodies : 1];  // second moments of the cells
    short4 child[kMomentBodies];    // nodes
    int parent[kMomentBodies];      // in the block's numbering
    int nint[kMomentBodies];        // kOutside: the cell reaches beyond the block
    int arrived[kMomentBodies];
    short ready[2][kMomentBodies];  // cells whose children are done, this round's and the next
    short tops[kMomentBodies];      // roots of the block's subtrees
    int nready[2], ntops;
};

template <bool kSplit, bool kSecond>
__global__ void __launch_bounds__(kMomentThreads, 2)
tree_moments(DeviceScalars* s, const double2* pos,
             const double* mass, int n, Tree t, Batch bt, float accept_scale,
             unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MomentSmem<kSecond>& S = *reinterpret_cast<MomentSmem<kSecond>*>(smem_raw);
    const int cells = s->cells;
    const int b0 = blockIdx.x * kMomentBodies, b1 = min(n, b0 + kMomentBodies);  // bodies [b0, b1)
    const int id0 = cell_id(t, b0);
    const int count = (b1 < n ? cell_id(t, b1) : cells) - id0;  // fewer than the bodies
    for (int k = threadIdx.x; k < b1 - b0; k += kMomentThreads) {
        const int b = b0 + k;
        const double2 p = pos[b];
        double3 v = make_double3(mass[b], p.x, p.y);
        // (leaf_last and the buckets mean something at leaf starts only, and
        // only these are read)
        if (t.leaf_last[b] != b) v = bucket_leaf(t, b);
        S.m[kMomentBodies + k] = v.x;
        S.x[kMomentBodies + k] = v.y;
        S.y[kMomentBodies + k] = v.z;
    }
    if (threadIdx.x == 0) {
        S.nready[0] = S.nready[1] = S.ntops = 0;
        S.m[kMomentNodes - 1] = S.x[kMomentNodes - 1] = S.y[kMomentNodes - 1] = 0.0;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += kMomentThreads) {
        const int2 r = t.range[id0 + k];
        const int nint = t.nint[id0 + k];
        const int4 ch = t.child[id0 + k];
        const bool own = r.x >= b0 && r.y < b1;
        auto node = [&](int ref) {
            return (short)(ref == INT_MIN ? kMomentNodes - 1
                           : ref >= 0     ? ref - id0
                                          : kMomentBodies + ~ref - b0);
        };
        if (own) S.child[k] = make_short4(node(ch.x), node(ch.y), node(ch.z), node(ch.w));
        S.nint[k] = own ? nint : kOutside;
        S.arrived[k] = 0;
        S.parent[k] = t.parent[id0 + k] - id0;
        if (nint == 0) {
            if (own) S.ready[0][atomicAdd(&S.nready[0], 1)] = (short)k;
            else S.tops[atomicAdd(&S.ntops, 1)] = (short)k;
        }
    }
    __syncthreads();
    auto own_cell = [&](int k) { return k >= 0 && k < count && S.nint[k] != kOutside; };
    // one of the block's own cells
    auto own_moments = [&](int k) {
        const short4 ch = S.child[k];
        const int node[4] = {ch.x, ch.y, ch.z, ch.w};
        double3 c[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = make_double3(S.m[node[q]], S.x[node[q]], S.y[node[q]]);
        const Moments o = combine_children<kSecond>(c, [&](int q) {
            const bool cell = kSecond && node[q] < kMomentBodies;
            return cell ? make_double3(S.s[0][node[q]], S.s[1][node[q]], S.s[2][node[q]])
                        : make_double3(0.0, 0.0, 0.0);
        });
        S.m[k] = o.m;
        S.x[k] = o.x;
        S.y[k] = o.y;
        if (kSecond) {
            S.s[0][k] = o.sxx;
            S.s[1][k] = o.sxy;
            S.s[2][k] = o.syy;
        }
    };
    // a cell whose children's moments are in global memory
    auto any_moments = [&](int id, int4 ch) {
        const int refs[4] = {ch.x, ch.y, ch.z, ch.w};
        double3 c[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = refs[q];
            c[q] = make_double3(0.0, 0.0, 0.0);
            if (r == INT_MIN) continue;
            if (r >= 0) {
                const double2 p = __ldcg(t.com + r);
                c[q] = make_double3(__ldcg(t.mass + r), p.x, p.y);
            } else {
                const double2 p = pos[~r];
                c[q] = make_double3(mass[~r], p.x, p.y);
                if (t.leaf_last[~r] != ~r) c[q] = bucket_leaf(t, ~r);
            }
        }
        const Moments o = combine_children<kSecond>(c, [&](int q) {
            if (refs[q] < 0) return make_double3(0.0, 0.0, 0.0);
            const double2* sc = reinterpret_cast<const double2*>(t.s64 + refs[q]);
            const double2 s01 = __ldcg(sc), s2 = __ldcg(sc + 1);
            return make_double3(s01.x, s01.y, s2.x);
        });
        store_moments<kSplit, kSecond>(id, o, true, s, pos, t, bt, accept_scale);
    };
    // Rounds: the cells that are ready are computed by consecutive threads (a
    // thread that climbed alone would leave its warp's other lanes idle), and
    // the last child to be done makes its parent ready for the next round.
    // Global memory is left out of the rounds, which follow one another.
    for (int r = 0;; ++r) {
        const int todo = S.nready[r & 1];
        if (todo == 0) break;
        for (int j = threadIdx.x; j < todo; j += kMomentThreads) {
            const int k = S.ready[r & 1][j];
            own_moments(k);
            const int p = S.parent[k];
            if (!own_cell(p)) {
                S.tops[atomicAdd(&S.ntops, 1)] = (short)k;
            } else if (atomicAdd(&S.arrived[p], 1) == S.nint[p] - 1) {
                S.ready[(r & 1) ^ 1][atomicAdd(&S.nready[(r & 1) ^ 1], 1)] = (short)p;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) S.nready[r & 1] = 0;
        __syncthreads();
    }
    for (int k = threadIdx.x; k < count; k += kMomentThreads)
        if (S.nint[k] != kOutside)
            store_moments<kSplit, kSecond>(
                id0 + k,
                Moments{S.m[k], S.x[k], S.y[k], kSecond ? S.s[0][k] : 0.0, kSecond ? S.s[1][k] : 0.0,
                        kSecond ? S.s[2][k] : 0.0},
                !own_cell(S.parent[k]), s, pos, t, bt, accept_scale);
    __syncthreads();
    // Beyond the block: the cells that reach out of it and have no internal
    // children, and the parents of the block's subtrees.  A path to the root
    // crosses at most 30 cells; the bound only guards against a malformed tree.
    const int ntops = S.ntops;
    for (int j = threadIdx.x; j < ntops; j += kMomentThreads) {
        const int k = S.tops[j];
        if (S.nint[k] == kOutside) any_moments(id0 + k, t.child[id0 + k]);
        int par = S.parent[k] + id0;
        for (int hop = 0; par >= 0; ++hop) {
            if (par >= cells || hop > kMaxLevel + 1) {
                atomicOr(&s->error, kErrTree);
                break;
            }
            const int needed = t.nint[par], up = t.parent[par];
            const int4 ch = t.child[par];
            if (arrive_acq_rel(t.ready + par) != needed - 1) break;
            t.ready[par] = 0;  // all have arrived: the learned features count again
            any_moments(par, ch);
            par = up;
        }
    }
}

// ---- SPLIT monopole moments from prefix sums ----------------------------
// A cell's bodies are one contiguous range of the sorted bodies, so its mass
// and first moment are differences of prefix sums over the bodies: one scan
// and one independent pass over the cells replace the bottom-up climb.  The
// sums are taken relative to each body's frame centre in FP64, so the
// cancellation in a difference stays far below the FP32 rounding of the cell
// records.  The FP64 parity mode (the reference's summation order) and the
// second and third moments (whose differences would cancel) keep the climb.
__device__ __forceinline__ double4 d4_add(double4 a, double4 b) {
    return make_double4(a.x + b.x, a.y + b.y, a.z + b.z, 0.0);
}

__device__ __forceinline__ double4 body_term(const double2* __restrict__ pos,
                                             const double* __restrict__ mass,
                                             const DeviceScalars* __restrict__ s, const Batch& bt,
                                             int i) {
    const double m = mass[i];
    const double2 p = pos[i], c = frame_center(s, bt, i);
    return make_double4(m, m * (p.x - c.x), m * (p.y - c.y), 0.0);
}

__device__ double4 block_sum_d4(double4 v, double4* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(kFull, v.x, o);
        v.y += __shfl_down_sync(kFull, v.y, o);
        v.z += __shfl_down_sync(kFull, v.z, o);
    }
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double4 tot = make_double4(0.0, 0.0, 0.0, 0.0);
    if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w) tot = d4_add(tot, red[w]);
    return tot;  // valid in thread 0
}

// Bodies of a tile are read in coalesced rows: each warp takes consecutive rows
// of 32.
constexpr int kWarpItems = 32 * kScanItems;
// Up to this many tiles a block of the second phase scans the totals itself
// (one warp, 8 per lane) instead of a kernel between the phases.
constexpr int kFewSums = 32 * kScanItems;

// Inclusive scan across the warp of the three components body_term fills.
__device__ __forceinline__ double4 warp_inclusive_d4(double4 v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(kFull, v.x, o);
        const double y = __shfl_up_sync(kFull, v.y, o);
        const double z = __shfl_up_sync(kFull, v.z, o);
        if (lane >= o) {
            v.x += x;
            v.y += y;
            v.z += z;
        }
    }
    return v;
}

// Exclusive scan, in thread order, of one value per thread of the block.
__device__ double4 block_exclusive_d4(double4 v, double4* part, double4& total) {
    part[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < kThreads; o <<= 1) {
        const double4 t = threadIdx.x >= o ? part[threadIdx.x - o] : make_double4(0.0, 0.0, 0.0, 0.0);
        __syncthreads();
        part[threadIdx.x] = d4_add(part[threadIdx.x], t);
        __syncthreads();
    }
    total = part[kThreads - 1];
    const double4 ex = threadIdx.x > 0 ? part[threadIdx.x - 1] : make_double4(0.0, 0.0, 0.0, 0.0);
    __syncthreads();  // part[] is reused by the caller's next round
    return ex;
}

// Many tiles: exclusive scan of the totals (one block, chunks of kThreads *
// kScanItems tiles in order); tiles[ntiles] = the grand total.
__global__ void __launch_bounds__(kThreads)
prefix_tiles_scan(double4* tiles, int ntiles) {
    chain_begin();
    __shared__ double4 part[kThreads];
    double4 carry = make_double4(0.0, 0.0, 0.0, 0.0);
    for (int c0 = 0; c0 < ntiles; c0 += kThreads * kScanItems) {
        const int base = c0 + threadIdx.x * kScanItems;
        double4 v[kScanItems];
        double4 run = make_double4(0.0, 0.0, 0.0, 0.0);
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = base + k < ntiles ? tiles[base + k] : make_double4(0.0, 0.0, 0.0, 0.0);
            run = d4_add(run, v[k]);
        }
        double4 total;
        double4 acc = d4_add(carry, block_exclusive_d4(run, part, total));
        for (int k = 0; k < kScanItems; ++k) {
            if (base + k < ntiles) tiles[base + k] = acc;
            acc = d4_add(acc, v[k]);
        }
        carry = d4_add(carry, total);
    }
    if (threadIdx.x == 0) tiles[ntiles] = carry;
}

// Phase 1: per tile of kScanTile bodies, the total.
__global__ void __launch_bounds__(kThreads)
prefix_reduce(const double2* pos, const double* mass, int n,
              const DeviceScalars* s, Batch bt, double4* tiles,
              unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    __shared__ double4 red[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int base = blockIdx.x * kScanTile + warp * kWarpItems + lane;
    double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + 32 * k < n) v = d4_add(v, body_term(pos, mass, s, bt, base + 32 * k));
    const double4 tot = block_sum_d4(v, red);
    if (threadIdx.x == 0) tiles[blockIdx.x] = tot;
}

// Phase 2: prefix[i] = sum over bodies before i; prefix[n] = the total.
// Each row of 32 bodies is scanned with shuffles; the rows' totals carry
// within the warp, and the warps' totals (one barrier) within the tile.  Few
// tiles (kFew): the block scans the tiles' totals itself.
// A warp of its own does that beside the rows' scans.
template <bool kFew>
// (four blocks per SM, 64 registers: 300k bodies 14.5 -> 12.0 us, 4M as with 80)
__global__ void __launch_bounds__(kThreads + (kFew ? 32 : 0), kFew ? 1 : 4)
prefix_apply(const double2* pos, const double* mass, int n,
             const DeviceScalars* s, Batch bt, const double4* tiles,
             int ntiles, double4* prefix) {
    chain_begin();
    __shared__ double4 wtot[kThreads / 32], tile_off;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int base = blockIdx.x * kScanTile + warp * kWarpItems + lane;
    const double4 zero = make_double4(0.0, 0.0, 0.0, 0.0);
    double4 ex[kScanItems];   // exclusive prefix within the row, then within the warp
    double4 carry = zero;     // total of the rows before
    if (!kFew || warp < kThreads / 32) {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            const int i = base + 32 * k;
            const double4 v = i < n ? body_term(pos, mass, s, bt, i) : zero;
            const double4 inc = warp_inclusive_d4(v);
            double4 e;
            e.x = __shfl_up_sync(kFull, inc.x, 1);
            e.y = __shfl_up_sync(kFull, inc.y, 1);
            e.z = __shfl_up_sync(kFull, inc.z, 1);
            e.w = 0.0;
            if (lane == 0) e = zero;
            ex[k] = d4_add(carry, e);
            const double4 row = make_double4(__shfl_sync(kFull, inc.x, 31), __shfl_sync(kFull, inc.y, 31),
                                             __shfl_sync(kFull, inc.z, 31), 0.0);
            carry = d4_add(carry, row);
        }
        if (lane == 0) wtot[warp] = carry;
    } else {
        // the scan kernel's sums, association included: lane l adds up tiles
        // 8 l .. 8 l + 7, the lanes are scanned, the tile's own lane goes on
        double4 v[kScanItems], run = zero;
        for (int k = 0; k < kScanItems; ++k) {
            const int q = lane * kScanItems + k;
            v[k] = q < ntiles ? tiles[q] : zero;
            run = d4_add(run, v[k]);
        }
        const double4 inc = warp_inclusive_d4(run);
        double4 acc;
        acc.x = __shfl_up_sync(kFull, inc.x, 1);
        acc.y = __shfl_up_sync(kFull, inc.y, 1);
        acc.z = __shfl_up_sync(kFull, inc.z, 1);
        acc.w = 0.0;
        if (lane == 0) acc = zero;
        if (lane == (int)blockIdx.x / kScanItems) {
            for (int k = 0; k < (int)blockIdx.x % kScanItems; ++k) acc = d4_add(acc, v[k]);
            tile_off = acc;
        }
        if (lane == 31 && blockIdx.x == ntiles - 1) prefix[n] = inc;
    }
    __syncthreads();
    if (kFew && warp == kThreads / 32) return;
    double4 off = kFew ? tile_off : tiles[blockIdx.x];
    for (int w = 0; w < warp; ++w) off = d4_add(off, wtot[w]);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + 32 * k;
        if (i < n) prefix[i] = d4_add(off, ex[k]);
    }
    if (!kFew && blockIdx.x == ntiles - 1 && threadIdx.x == 0) prefix[n] = tiles[ntiles];
}

__device__ void cell_from_prefix(const double4* __restrict__ prefix, const Tree& t,
                                 const DeviceScalars* __restrict__ s, const Batch& bt,
                                 const double2* __restrict__ pos, int id, int2 r, int level,
                                 float accept_scale) {
    const double4 a = prefix[r.x], b = prefix[r.y + 1];
    const double M = b.x - a.x;
    const double rx = (b.y - a.y) / M, ry = (b.z - a.z) / M;
    const double2 fc = frame_center(s, bt, r.x);
    const double2 com = make_double2(fc.x + rx, fc.y + ry);
    t.mass[id] = M;
    t.com[id] = com;
    t.cell4[id] = make_float4((float)rx, (float)ry, (float)M,
                              accept_size2(s, bt, pos, r.x, level, com, accept_scale));
}


// ---- learned features: second and third moments -------------------------
// The features need S and T about each cell's centre of mass, which the
// prefix pass has already written.  A cell with fewer than kDirectCell
// bodies, or with only leaf children, sums them directly over its bodies;
// a larger cell combines its children by the parallel-axis shift
//   S = sum_c [S_c + m_c d d^T]
//   T = sum_c [T_c + (d_i S_c,jk + d_j S_c,ik + d_k S_c,ij) + m_c d_i d_j d_k],
// bottom-up: a directly summed cell under a larger parent arrives at the
// parent's counter, and the last child to arrive computes the parent and
// climbs on.  Only the few cells above the direct size climb.  FP32: the
// moments only feed BF16 features.
constexpr int kDirectCell = 32;

__device__ __forceinline__ bool direct_cell(const Tree& t, int id) {
    const int2 r = t.range[id];
    return r.y - r.x < kDirectCell || t.nint[id] == 0;
}

__device__ __forceinline__ double child_mass(const Tree& t, const double* __restrict__ mass,
                                             int r) {
    if (r >= 0) return t.mass[r];
    const int b = ~r;
    return t.leaf_last[b] == b ? mass[b] : t.bucket_mass[b];
}

// The cell's feature record (the BF16 features, then COM, mass and width)
// and its S and T for the parent's shift.
__device__ void write_features(const Tree& t, const DeviceScalars* __restrict__ s,
                               const Batch& bt, const double* __restrict__ mass, int id,
                               const float* S, const float* T) {
    const int4 ch = t.child[id];
    const int refs[4] = {ch.x, ch.y, ch.z, ch.w};
    double mmax = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (refs[q] != INT_MIN) mmax = fmax(mmax, child_mass(t, mass, refs[q]));
    const double M = t.mass[id];
    const int first = t.range[id].x;
    const double w2 = cell_width2(s, bt, first, t.level[id]), w = sqrt(w2);
    const float im2 = (float)(1.0 / (M * w2)), im3 = (float)(1.0 / (M * w2 * w));
    __stcg(t.s32 + id, make_float4(S[0], S[1], S[2], 0.f));
    __stcg(t.t32 + id, make_float4(T[0], T[1], T[2], T[3]));
    const float4 c4 = t.cell4[id];
    t.cellh[2 * id] = make_uint4(bf16_pair((float)(mmax / M), S[0] * im2),
                                 bf16_pair(S[1] * im2, S[2] * im2),
                                 bf16_pair(T[0] * im3, T[1] * im3),
                                 bf16_pair(T[2] * im3, T[3] * im3));
    t.cellh[2 * id + 1] = make_uint4(__float_as_uint(c4.x), __float_as_uint(c4.y),
                                     __float_as_uint(c4.z), __float_as_uint((float)w));
}

// One mass point (or a child's moments) at offset (dx, dy) from the COM.
__device__ __forceinline__ void add_shifted(float m, float dx, float dy, const float4 cs,
                                            const float4 ct, float* S, float* T) {
    T[0] += ct.x + 3.f * dx * cs.x + m * dx * dx * dx;
    T[1] += ct.y + 2.f * dx * cs.y + dy * cs.x + m * dx * dx * dy;
    T[2] += ct.z + dx * cs.z + 2.f * dy * cs.y + m * dx * dy * dy;
    T[3] += ct.w + 3.f * dy * cs.z + m * dy * dy * dy;
    S[0] += cs.x + m * dx * dx;
    S[1] += cs.y + m * dx * dy;
    S[2] += cs.z + m * dy * dy;
}

// A block deals its cells to its threads by size, so that the lanes of a warp
// sum over about as many bodies each (in id order 9 of 32 lanes were active).
__global__ void __launch_bounds__(kThreads)
learned_features(DeviceScalars* s, const double2* pos,
                 const double* mass, Tree t, Batch bt) {
    chain_begin();
    const int id0 = blockIdx.x * blockDim.x;
    const int cells = s->cells;
    if (id0 >= cells) return;
    __shared__ int bin[kDirectCell + 1];  // sizes of more than 32 bodies, 32, 31, ..., 1
    __shared__ short deal[kThreads];
    for (int k = threadIdx.x; k <= kDirectCell; k += kThreads) bin[k] = 0;
    __syncthreads();
    int id = id0 + threadIdx.x;
    const bool mine = id < cells && direct_cell(t, id);
    int rank = 0, b = 0;
    if (mine) {
        const int2 r = t.range[id];
        b = kDirectCell - min(r.y - r.x, kDirectCell);
        rank = atomicAdd(&bin[b], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // where each size starts (size 1 has no cells)
        const int inc = warp_inclusive(bin[threadIdx.x]);
        bin[threadIdx.x] = inc - bin[threadIdx.x];
        if (threadIdx.x == 31) bin[kDirectCell] = inc;
    }
    __syncthreads();
    if (mine) deal[bin[b] + rank] = (short)threadIdx.x;
    __syncthreads();
    if ((int)threadIdx.x >= bin[kDirectCell]) return;
    id = id0 + deal[threadIdx.x];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    {
        const double2 com = t.com[id];
        const int2 r = t.range[id];
        float S[3] = {0.f, 0.f, 0.f}, T[4] = {0.f, 0.f, 0.f, 0.f};
        for (int j = r.x; j <= r.y; ++j) {
            const double2 p = pos[j];
            add_shifted((float)mass[j], (float)(p.x - com.x), (float)(p.y - com.y), zero, zero, S,
                        T);
        }
        write_features(t, s, bt, mass, id, S, T);
    }
    // A path to the root crosses at most 30 cells; the bound only guards
    // against a malformed tree.
    for (int hop = 0;; ++hop) {
        const int par = t.parent[id];
        if (par < 0) return;
        if (par >= cells || hop > kMaxLevel + 1) {
            atomicOr(&s->error, kErrTree);
            return;
        }
        if (direct_cell(t, par)) return;  // its own thread sums it
        const int arrived = arrive_acq_rel(t.ready + par);
        if (arrived != t.nint[par] - 1) return;
        id = par;
        const double2 com = t.com[id];
        const int4 ch = t.child[id];
        const int refs[4] = {ch.x, ch.y, ch.z, ch.w};
        float S[3] = {0.f, 0.f, 0.f}, T[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = refs[q];
            if (r == INT_MIN) continue;
            double2 cc;
            float4 cs = zero, ct = zero;
            if (r >= 0) {
                cc = t.com[r];
                cs = __ldcg(t.s32 + r);
                ct = __ldcg(t.t32 + r);
            } else {
                const int b = ~r;
                cc = t.leaf_last[b] == b ? pos[b] : t.bucket_com[b];
            }
            add_shifted((float)child_mass(t, mass, r), (float)(cc.x - com.x), (float)(cc.y - com.y),
                        cs, ct, S, T);
        }
        write_features(t, s, bt, mass, id, S, T);
    }
}

// ---- SPLIT target groups -----------------------------------------------
// A cell with more than gsize bodies hands its small children (cells or
// leaves with <= gsize bodies) to groups: consecutive small children are
// merged while the sum stays <= gsize, so a group never leaves its parent
// cell and its bounding box stays within one cell width.  With fill set, a
// child that would overflow the group is split instead: the group takes
// exactly gsize bodies and the child's rest starts the next group.  Multi-body
// leaves larger than a group are cut into chunks of gsize.  kWrite = false
// counts the groups of each cell, kWrite = true writes them.
//
// Children in key order are quadrants 0..3; 0,1 and 2,3 are the two halves of
// the cell, while a run that takes quadrants from both halves has the whole
// cell as its bounding box.  When one child is large (it emits its own
// groups), such a box would cover that dense quadrant and the group's walk
// would open it down to its bodies: in a sparse disc tail, a group of outer
// bodies then walked the whole core on one warp (2.3 ms of a 65,536-body
// step).  So with a large child present, runs also end at the half boundary.
// The groups of one cell with body range rg and nc children in code order
// ([ca, cb], leaf marks the leaf children); returns their counts and, with kWrite,
// writes them from out on, those of up to `small` bodies from out_small on.
template <bool kWrite>
__device__ __forceinline__ int cell_groups(int2 rg, bool is_root, int nc, const int* ca, const int* cb,
                           const bool* leaf, int gsize, int fill, int small, const Batch& bt,
                           const uint64_t* __restrict__ key, int2* __restrict__ out,
                           int2* __restrict__ out_small) {
    int emitted = 0;
    auto emit = [&](int a, int b) {
        const bool is_small = b - a < small;
        if (kWrite) *(is_small ? out_small++ : out++) = make_int2(a, b);
        emitted += small > 0 ? (1 << kSmallBits) + is_small : 1;
    };
    // batched universes: a forest cell above the universe roots may hold few
    // bodies but never becomes a group; it hands its children on instead
    const bool spans = bt.nuni && bt.uid[rg.x] != bt.uid[rg.y];
    if (rg.y - rg.x + 1 <= gsize && !spans) {
        if (is_root) emit(rg.x, rg.y);  // the whole (small) tree is one group
        return emitted;
    }
    bool large = false;  // some child emits its own groups
#pragma unroll
    for (int q = 0; q < 4; ++q)
        large |= q < nc && (cb[q] - ca[q] + 1 > gsize || (bt.nuni && bt.uid[ca[q]] != bt.uid[cb[q]]));
    // the children differ in digit `level` of their codes; its high bit is
    // the half (read only when a large child makes it matter)
    const int level = large ? min(lcp_digits(key[rg.x], key[rg.y]), 31) : 0;
    int run_a = -1, run_b = -1, run_half = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= nc) continue;
        const int a = ca[q], b = cb[q];
        const int cnt = b - a + 1;
        if (cnt > gsize || (bt.nuni && bt.uid[a] != bt.uid[b])) {  // the child emits
            if (run_a >= 0) emit(run_a, run_b);
            run_a = -1;
            if (leaf[q])  // oversized multi-body leaf: chunks of one group each
                for (int k = a; k <= b; k += gsize) emit(k, min(b, k + gsize - 1));
            continue;
        }
        const int half = large ? (int)(key[a] >> (63 - 2 * level)) & 1 : 0;
        // a group never spans two universes (a forest cell's children may),
        // nor both halves of a cell that has a large child
        if (run_a >= 0 && ((bt.nuni && bt.uid[a] != bt.uid[run_a]) ||
                           (large && half != run_half))) {
            emit(run_a, run_b);
            run_a = -1;
        } else if (run_a >= 0 && b - run_a + 1 > gsize) {
            if (fill) {
                // fill the group; the rest of this child starts the next one
                emit(run_a, run_a + gsize - 1);
                run_a += gsize;
                run_b = b;
                continue;
            }
            emit(run_a, run_b);
            run_a = -1;
        }
        if (run_a < 0) {
            run_a = a;
            run_half = half;
        }
        run_b = b;
    }
    if (run_a >= 0) emit(run_a, run_b);
    return emitted;
}

// Writes the groups, which the linking pass counted, one block per tile: the
// tile's counts are scanned (each warp 8 rows of 32 cells), and the few cells
// that have groups (1.5% at 4M) are listed and written one thread each.
constexpr int kCellBits = 11;
constexpr int kSmallMask = (1 << kSmallBits) - 1;
static_assert(kAnsvTile <= 1 << kCellBits && kCellBits + kSmallBits < 31, "a list word's fields");

template <bool kSmall>  // small groups are listed apart
__global__ void __launch_bounds__(kThreads, kSmall ? 4 : 5)
tree_groups_write(int n, int gsize, int fill, int small, Tree t, DeviceScalars* s,
                  Batch bt, const uint64_t* key, unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    const int tile = blockIdx.x;
    if (s->cells == 0) {  // no cell: the root leaf holds all bodies
        const int ng = (n + gsize - 1) / gsize;
        for (int k = tile * kThreads + threadIdx.x; k < ng; k += gridDim.x * kThreads)
            t.groups[k] = make_int2(k * gsize, min(n, (k + 1) * gsize) - 1);
        if (tile == 0 && threadIdx.x == 0) s->groups = ng;
        return;
    }
    __shared__ int2 wsum[kThreads / 32], wbefore[kThreads / 32];
    __shared__ int wlarge[kThreads / 32];
    // cells with groups: {cell and small groups before (kCellBits), others before}
    __shared__ int2 some[kAnsvTile];
    __shared__ int nsome;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int count = t.tile_count[tile], id0 = t.tile_cells[tile];
    if (threadIdx.x == 0) nsome = 0;
    // the groups of the tiles before, and all large ones (8 loads per thread at
    // 4M; a scan by the linking pass's last block cost its other blocks more in
    // fences)
    int before = 0, before_small = 0, large = 0;
#pragma unroll 4
    for (int q = threadIdx.x; q < (kSmall ? (int)gridDim.x : tile); q += kThreads) {
        const int g = t.tile_groups[q];
        const int sm = kSmall ? g & kSmallMask : 0, lg = kSmall ? (g >> kSmallBits) - sm : g;
        large += lg;
        before += q < tile ? lg : 0;
        before_small += q < tile ? sm : 0;
    }
    // the tile's counts: large groups, small ones
    int v[kAnsvItems];
    int2 ex[kAnsvItems], carry = make_int2(0, 0);
#pragma unroll
    for (int k = 0; k < kAnsvItems; ++k) {
        const int j = (warp * kAnsvItems + k) * 32 + lane;
        v[k] = j < count ? t.gcount[id0 + j] : 0;
    }
#pragma unroll
    for (int k = 0; k < kAnsvItems; ++k) {
        const int sm = kSmall ? v[k] & kSmallMask : 0;
        const int lg = kSmall ? (v[k] >> kSmallBits) - sm : v[k];
        const int il = warp_inclusive(lg), is = kSmall ? warp_inclusive(sm) : 0;
        ex[k] = make_int2(carry.x + il - lg, carry.y + is - sm);
        carry.x += __shfl_sync(kFull, il, 31);
        if (kSmall) carry.y += __shfl_sync(kFull, is, 31);
    }
    before = __reduce_add_sync(kFull, before);
    if (kSmall) {
        before_small = __reduce_add_sync(kFull, before_small);
        large = __reduce_add_sync(kFull, large);
    }
    if (lane == 0) {
        wsum[warp] = carry;
        wbefore[warp] = make_int2(before, before_small);
        wlarge[warp] = large;
    }
    __syncthreads();
    int2 off = make_int2(0, 0), in_tile = make_int2(0, 0);  // (small ones follow all others)
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        off.x += wbefore[w].x;
        off.y += wlarge[w] + wbefore[w].y;
        in_tile.x += w < warp ? wsum[w].x : 0;
        in_tile.y += w < warp ? wsum[w].y : 0;
    }
    if (tile == gridDim.x - 1 && threadIdx.x == kThreads - 1)
        s->groups = kSmall ? off.y + in_tile.y + carry.y : off.x + in_tile.x + carry.x;
#pragma unroll
    for (int k = 0; k < kAnsvItems; ++k)
        if (v[k])
            some[atomicAdd(&nsome, 1)] =
                make_int2((warp * kAnsvItems + k) * 32 + lane | (in_tile.y + ex[k].y) << kCellBits,
                          in_tile.x + ex[k].x);
    __syncthreads();
    for (int q = threadIdx.x; q < nsome; q += kThreads) {
        const int id = id0 + (some[q].x & (1 << kCellBits) - 1);
        const int2 rg = t.range[id];
        const int4 ch = t.child[id];
        const int refs[4] = {ch.x, ch.y, ch.z, ch.w};
        int ca[4], cb[4], nc = 0;
        bool leaf[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int r = refs[c];
            if (r == INT_MIN) break;
            leaf[c] = r < 0;
            if (r >= 0) {
                const int2 cr = t.range[r];
                ca[c] = cr.x;
                cb[c] = cr.y;
            } else {
                ca[c] = ~r;
                cb[c] = t.leaf_last[ca[c]];
            }
            nc = c + 1;
        }
        cell_groups<true>(rg, id == s->root, nc, ca, cb, leaf, gsize, fill, kSmall ? small : 0, bt, key,
                          t.groups + off.x + some[q].y,
                          t.groups + off.y + (some[q].x >> kCellBits));
    }
}

// Root reference of each universe: the cell whose body range is exactly the
// universe's (found like a child cell in tree_link), or its single leaf.
__global__ void batch_roots(const uint64_t* key, Tree t, Batch bt) {
    chain_begin();
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= bt.nuni) return;
    const int a = bt.off[u], b = bt.off[u + 1] - 1;
    if (b <= a) {
        bt.root[u] = ~a;
        return;
    }
    const int c = lcp_digits(key[a], key[b]);
    if (c >= kMaxLevel) {  // all bodies of the universe in one level-30 leaf
        bt.root[u] = ~a;
        return;
    }
    bt.root[u] = cell_id(t, gallop_right(key, a, b, c + 1));
}

inline unsigned blocks_for(int64_t n, int threads) {
    return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

void launch_batch_roots(nb_ctx* c) {
    if (c->batch.nuni == 0) return;
    c->launches += 1;
    chain_launch(c->stream, true, batch_roots, blocks_for(c->batch.nuni, 128), 128, 0, 1,
                 c->sort.key[0], c->tree, c->batch);
}

static int small_group(const nb_ctx* c) {
    const int gsize = split_group_size(c);
    return c->n <= kSmallLastMax && gsize > 32 && !(c->p.flags & NB_FLAG_LEARNED) ? gsize / 2 : 0;
}

void launch_groups(nb_ctx* c) {
    c->launches += 1;
    // plain SPLIT fills groups to gsize bodies across sibling cells (fuller
    // warps, measured 2.6% off the walk at 4M with slightly lower errors); the
    // learned correction keeps groups of whole cells, whose residuals it fits.
    const int fill = (c->p.flags & NB_FLAG_LEARNED) ? 0 : 1;
    const int small = small_group(c);
    chain_launch(c->stream, true, small > 0 ? tree_groups_write<true> : tree_groups_write<false>,
                 blocks_for(c->n, kAnsvTile), kThreads, 0, 1, (int)c->n, split_group_size(c), fill,
                 small, c->tree, c->scal, c->batch, c->sort.key[0],
                 mark_of(c, 6));
}

// SPLIT without quadrupoles takes its monopoles from prefix sums over the
// sorted bodies, which the linking pass turns into cell records.
static bool mono_prefix(const nb_ctx* c) {
    return c->p.mode == NB_MODE_SPLIT && !(c->p.flags & NB_FLAG_QUADRUPOLE);
}

// The acceptance-size factor of the b_max test (0 = plain width test).
static float split_accept_scale(const nb_ctx* c) {
    const double ratio = c->p.bmax_ratio;
    return c->p.mode == NB_MODE_SPLIT && ratio > 0.0
               ? (float)(c->p.theta * c->p.theta / (ratio * ratio))
               : 0.f;
}

void launch_prefix_sums(nb_ctx* c, const BodyBuffers& b) {
    if (!mono_prefix(c)) return;
    const int n = (int)c->n, ptiles = (int)blocks_for(n, kScanTile);
    const bool few = ptiles <= kFewSums;
    c->launches += few ? 2 : 3;
    chain_launch(c->stream, true, prefix_reduce, ptiles, kThreads, 0, 1, b.pos, b.mass, n, c->scal,
                 c->batch, c->tree.prefix_tiles, mark_of(c, 3));
    if (!few)
        chain_launch(c->stream, true, prefix_tiles_scan, 1, kThreads, 0, 1, c->tree.prefix_tiles,
                     ptiles);
    chain_launch(c->stream, true, few ? prefix_apply<true> : prefix_apply<false>, ptiles,
                 kThreads + (few ? 32 : 0), 0, 1, b.pos, b.mass, n, c->scal, c->batch, c->tree.prefix_tiles, ptiles,
                 c->tree.prefix);
}

void launch_tree(nb_ctx* c, const BodyBuffers& b) {
    const int n = (int)c->n;
    const bool mono = mono_prefix(c);
    const uint64_t* key = c->sort.key[0];
    Tree& t = c->tree;
    const int tiles = (int)blocks_for(n, kAnsvTile);
    const bool few = tiles <= kFewTiles;
    c->launches += few ? 3 : 4;
    const TileTable tab{t.ansv_first, t.ansv_last, few ? 1 : tiles, few ? kAnsvLevels : 1};
    const bool wide = tiles <= c->sm_count;
    chain_launch(c->stream, true, wide ? tree_lcp<kWideThreads> : tree_lcp<kThreads>, tiles,
                 wide ? kWideThreads : kThreads, 0, 1, key, n, t.lcp8, tab, c->scal->lcp_hist,
                 mark_of(c, 4));
    if (!few)
        chain_launch(c->stream, true, tree_ansv_tiles, kAnsvLevels, kTileScanThreads, 0, 1, tiles,
                     t.ansv_first, t.ansv_last);
    chain_launch(c->stream, true, wide ? tree_ansv<kWideThreads> : tree_ansv<kThreads>, tiles,
                 wide ? kWideThreads : kThreads, 0, 1, t, n, tiles, tab, c->scal);
    // SPLIT: the cells count their target groups as they link
    const int gsize = c->p.mode == NB_MODE_SPLIT ? split_group_size(c) : 0;
    const int fill = (c->p.flags & NB_FLAG_LEARNED) ? 0 : 1;
    chain_launch(c->stream, true, mono ? tree_link<true> : tree_link<false>, tiles * kLinkBlocks,
                 kThreads, 0, 1, key, n, b.pos, b.mass, t, c->scal, mono ? t.prefix : nullptr,
                 c->batch, mono ? split_accept_scale(c) : 0.f, gsize, fill,
                 gsize > 0 ? small_group(c) : 0);
}

void launch_features(nb_ctx* c, const BodyBuffers& b, bool chained) {
    const int cap = (int)(c->n > 1 ? c->n - 1 : 1);
    c->launches += 1;
    chain_launch(c->stream, chained, learned_features, blocks_for(cap, kThreads), kThreads, 0, 1, c->scal,
                 b.pos, b.mass, c->tree, c->batch);
}

template <bool kSplit, bool kSecond>
static void launch_climb(nb_ctx* c, const BodyBuffers& b, float accept_scale) {
    auto* kernel = tree_moments<kSplit, kSecond>;
    const size_t smem = sizeof(MomentSmem<kSecond>);
    c->launches += 1;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    chain_launch(c->stream, true, kernel, blocks_for(c->n, kMomentBodies), kMomentThreads, smem, 1,
                 c->scal, b.pos, b.mass, (int)c->n, c->tree, c->batch, accept_scale, mark_of(c, 5));
}

// SPLIT monopoles need none: the prefix sums ran before the tree, and the
// linking pass wrote every cell's record from them.
void launch_moments(nb_ctx* c, const BodyBuffers& b, bool split) {
    if (!split) launch_climb<false, false>(c, b, 0.f);
    else if (c->p.flags & NB_FLAG_QUADRUPOLE) launch_climb<true, true>(c, b, split_accept_scale(c));
}

}  // namespace nb
