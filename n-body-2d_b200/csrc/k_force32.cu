// k_force32.cu -- SPLIT mode: warp-cooperative group traversal in FP32 with
// shared-memory interaction lists, fused with the FP64 kick and drift.
//
// One warp owns a group of 32 Morton-consecutive bodies (one per lane) and
// walks the tree once for the whole group.  Each round the warp pops up to 32
// cells from its shared-memory stack, one per lane, and decides for each:
//   * accept: the cell does not hold a body of the group and
//     width^2 < theta^2 d^2, d = distance from the cell's centre of mass to
//     the group's bounding box (so every body of the group passes the
//     reference's per-body test width^2 < theta^2 d_i^2 of CU:463);
//     the cell joins the cell list;
//   * summed directly: a cell with at most leaf_size bodies, or a leaf; its
//     bodies join the body list;
//   * opened: its children are pushed.
// Whenever a list holds 32 entries, every lane sums them for its own body,
// reading entries by broadcast from shared memory.  Cells contribute their
// monopole (the reference's pair law, CU:427-431) and, with quadrupoles on,
// the second-moment term of the softened potential.  Accelerations
// accumulate in FP32; velocities and positions are updated in FP64.
#include <cfloat>
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nb_internal.cuh"

namespace nb {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerBlock = 4;
constexpr int kStk = 256;              // stack bound kept by the batch size rule
constexpr int kStkAlloc = kStk + 96;   // + one depth-first descent (<= 3 x 30 + 1)
constexpr int kList = 64;
constexpr int kBodiesPerLane = 2;      // group of 64 bodies per warp
constexpr int kDefaultLeaf = 8;        // cells this small are summed body by body
constexpr int kMaxBPL = 4;             // largest group: 128 bodies per warp

// Interaction lists hold entries in pairs, so that one lane evaluates two
// entries with the packed FP32x2 instructions of sm_100 (FADD2/FMUL2/FFMA2):
// pair k is xy[k] = (x0, x1, y0, y1) and m[k] = (m0, m1), with the quadrupole
// (xx0, xx1, xy0, xy1) in qa[k] and (yy0, yy1) in qb[k].
struct WarpLists {
    int stack[kStkAlloc];
    float4 cxy[kList / 2];
    float2 cm[kList / 2];
    float4 qa[kList / 2];
    float2 qb[kList / 2];
    float4 bxy[kList / 2];
    float2 bm[kList / 2];
    float2 tot[2 * kMaxBPL][32];   // running {x, y} sums of each lane's bodies (halves kept apart)
};

// An entry that adds nothing: zero mass far away, so that d2 stays finite
// and positive whatever eps2 is (it completes a pair at an odd count).
constexpr float kPadCoord = 1e15f;

// 1/sqrt(x) on the special-function unit.  kExact keeps subnormal x (the
// eps2 = 0 variant, where d2 can be that small); otherwise x >= eps2 is a
// normal float and the flush-to-zero form saves the subnormal handling.
template <bool kExact>
__device__ __forceinline__ float rsq(float x) {
    if (kExact) return rsqrtf(x);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void put_entry(float4* xy, float2* m, int slot, float x, float y,
                                          float mass) {
    float* f = reinterpret_cast<float*>(xy + (slot >> 1));
    f[slot & 1] = x;
    f[2 + (slot & 1)] = y;
    reinterpret_cast<float*>(m)[slot] = mass;
}

__device__ __forceinline__ int warp_exclusive_sum(int v, int& total) {
    const int lane = threadIdx.x & 31;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += t;
    }
    total = __shfl_sync(kFull, inc, 31);
    return inc - v;
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// One pair of list entries against the lane's kBPL bodies.  nx/ny hold the
// negated body coordinates broadcast to both halves.  Each half follows the
// scalar law d2 = dx^2 + (dy^2 + eps2), a = (m / r^2) / r of the reference's
// pair term (CU:427-431) with the same rounding; the halves are separate
// partial sums.  kZeroSoft: eps2 = 0, where an entry at the body's own FP32
// coordinates (the body itself, or one that coincides with it at FP32
// resolution) adds nothing instead of 0 * inf, and 1/sqrt keeps subnormal
// arguments.  With eps2 > 0 the body's own entry has dx = dy = 0 exactly and
// adds 0 without a test.
template <bool kZeroSoft, int kBPL>
__device__ __forceinline__ void mono_pair(const float4 xy, const float2 m, const float2* nx,
                                          const float2* ny, const float2 e2, float2* ax,
                                          float2* ay) {
    const float2 ex = make_float2(xy.x, xy.y), ey = make_float2(xy.z, xy.w);
#pragma unroll
    for (int b = 0; b < kBPL; ++b) {
        const float2 dx = __fadd2_rn(ex, nx[b]);
        const float2 dy = __fadd2_rn(ey, ny[b]);
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, e2));
        const float2 inv = make_float2(rsq<kZeroSoft>(d2.x), rsq<kZeroSoft>(d2.y));
        float2 a = __fmul2_rn(__fmul2_rn(m, __fmul2_rn(inv, inv)), inv);
        if (kZeroSoft) {
            a.x = d2.x == 0.f ? 0.f : a.x;
            a.y = d2.y == 0.f ? 0.f : a.y;
        }
        ax[b] = __ffma2_rn(dx, a, ax[b]);
        ay[b] = __ffma2_rn(dy, a, ay[b]);
    }
}

// Monopole plus the second-moment term of the softened potential,
//   a = d [M r^-3 - 1.5 tr(S) r^-5 + 7.5 (d.S.d) r^-7] - 3 r^-5 S d,
// from the cell record Q = 7.5 S (the moments pass stores it so) as
//   a = d r^-3 [M + r^-2 (-0.2 tr(Q) + r^-2 (d.Q.d))] - 0.4 r^-3 r^-2 Q d:
// 21 packed FMA-pipe operations per body and pair (23 in the textbook order).
// The walk is FMA-pipe bound with quadrupoles, so the count is the cost.
template <bool kZeroSoft, int kBPL>
__device__ __forceinline__ void quad_pair(const float4 xy, const float2 m, const float4 qa,
                                          const float2 qb, const float2* nx, const float2* ny,
                                          const float2 e2, float2* ax, float2* ay) {
    const float2 ex = make_float2(xy.x, xy.y), ey = make_float2(xy.z, xy.w);
    const float2 qxx = make_float2(qa.x, qa.y), qxy = make_float2(qa.z, qa.w), qyy = qb;
    const float2 tr = __fmul2_rn(make_float2(-0.2f, -0.2f), __fadd2_rn(qxx, qyy));
    const float2 m04 = make_float2(-0.4f, -0.4f);
#pragma unroll
    for (int b = 0; b < kBPL; ++b) {
        const float2 dx = __fadd2_rn(ex, nx[b]);
        const float2 dy = __fadd2_rn(ey, ny[b]);
        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, e2));
        const float2 inv = make_float2(rsq<kZeroSoft>(d2.x), rsq<kZeroSoft>(d2.y));
        const float2 inv2 = __fmul2_rn(inv, inv);
        const float2 inv3 = __fmul2_rn(inv, inv2);
        const float2 sdx = __ffma2_rn(qxx, dx, __fmul2_rn(qxy, dy));
        const float2 sdy = __ffma2_rn(qxy, dx, __fmul2_rn(qyy, dy));
        const float2 dsd = __ffma2_rn(dx, sdx, __fmul2_rn(dy, sdy));
        const float2 radial = __fmul2_rn(__ffma2_rn(__ffma2_rn(dsd, inv2, tr), inv2, m), inv3);
        const float2 k5 = __fmul2_rn(inv3, __fmul2_rn(m04, inv2));
        ax[b] = __ffma2_rn(dx, radial, __ffma2_rn(k5, sdx, ax[b]));
        ay[b] = __ffma2_rn(dy, radial, __ffma2_rn(k5, sdy, ay[b]));
    }
}

// Every kFoldFlushes list flushes, the lane's register sums are added to the
// body's running totals, kept in the warp's shared lists, and restart from
// zero (blocked summation): the FP32 rounding of a body's total then grows
// with the block length plus the number of blocks, not with the number of
// terms (a body's terms mostly share their sign, so a running sum's rounding
// adds up).  The totals live in shared memory so that the blocking costs no
// registers, and a block spans four flushes so that it costs few
// instructions.
constexpr int kFoldFlushes = 4;
template <int kBPL>
__device__ __forceinline__ void fold_block(WarpLists& L, float2* ax, float2* ay) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int b = 0; b < kBPL; ++b) {
        L.tot[2 * b][lane] = __fadd2_rn(L.tot[2 * b][lane], ax[b]);
        L.tot[2 * b + 1][lane] = __fadd2_rn(L.tot[2 * b + 1][lane], ay[b]);
        ax[b] = ay[b] = make_float2(0.f, 0.f);
    }
}

// Which entries a lane takes: pairs slot, slot + slots, ...  A lane for each
// body takes them all (slots = 1); where a block shares a group (kShare), a
// group of 16 or 8 bodies gives each 2 or 4 lanes, whose sums are added at the
// end.
struct Slots {
    int slot, slots;
};

// The first npairs pairs of the cell list (kCells) or the body list against
// the lane's first kN bodies.
template <bool kCells, bool kQuad, bool kZeroSoft, int kN>
__device__ __forceinline__ void sum_pairs(const WarpLists& L, int npairs, Slots sl, const float2* nx,
                                          const float2* ny, const float2 e2, float2* ax, float2* ay) {
    auto pair = [&](int k) {
        if (kCells && kQuad)
            quad_pair<kZeroSoft, kN>(L.cxy[k], L.cm[k], L.qa[k], L.qb[k], nx, ny, e2, ax, ay);
        else if (kCells)
            mono_pair<kZeroSoft, kN>(L.cxy[k], L.cm[k], nx, ny, e2, ax, ay);
        else
            mono_pair<kZeroSoft, kN>(L.bxy[k], L.bm[k], nx, ny, e2, ax, ay);
    };
    if (kN > 1) {
        if (npairs == 16) {
#pragma unroll 4
            for (int k = 0; k < 16; ++k) pair(k);
        } else {
            for (int k = 0; k < npairs; ++k) pair(k);
        }
    } else if (npairs == 16) {
        for (int k = sl.slot; k < 16; k += 4 * sl.slots) {
#pragma unroll
            for (int q = 0; q < 4; ++q) pair(k + q * sl.slots);
        }
    } else {
        for (int k = sl.slot; k < npairs; k += sl.slots) pair(k);
    }
}

// kBPL bodies per lane, or one where the group has no more bodies than lanes:
// a quarter of the groups of up to 64 bodies have 32 or fewer, and the pair
// terms of empty places were a sixth of all.
template <bool kCells, bool kQuad, bool kZeroSoft, int kBPL>
__device__ __forceinline__ void sum_list(WarpLists& L, int npairs, bool one, Slots sl,
                                         const float2* nx, const float2* ny, const float2 e2,
                                         float2* ax, float2* ay, bool fold) {
    if (kBPL == 1 || one)
        sum_pairs<kCells, kQuad, kZeroSoft, 1>(L, npairs, sl, nx, ny, e2, ax, ay);
    else
        sum_pairs<kCells, kQuad, kZeroSoft, kBPL>(L, npairs, sl, nx, ny, e2, ax, ay);
    if (fold) fold_block<kBPL>(L, ax, ay);
}

// Walk the tree for one group [g0, g1] of <= 32 kBPL bodies (lane l owns
// g0 + l, g0 + 32 + l, ...) and accumulate the FP32 accelerations.
// kShare: the block's warps walk for the same group.  Each opens the top of the
// tree until its stack holds kShareAt nodes, from which warp `part` then keeps
// every kWarpsPerBlock-th; what is accepted or summed directly before that counts
// in the first warp only.
constexpr int kShareAt = 24;
static_assert(kShareAt <= 32 && kWarpsPerBlock == 4, "a warp's part of the stack fits its lanes");

template <bool kQuad, int kBPL, bool kLearned, bool kZeroSoft, bool kShare>
__device__ __forceinline__ void walk_group(WarpLists& L, const Tree& t, int root, int n, int g0,
                                           int g1, bool one, Slots sl, const float* px,
                                           const float* py,
                                           const bool* act_body, float eps2, float theta2,
                                           int leaf_size, float* ax, float* ay,
                                           unsigned long long& ncell, unsigned long long& npair,
                                           unsigned* err, int* band, int& nband, int band_cap,
                                           float band2, int part) {
    const int lane = threadIdx.x & 31;
    float bx0 = INFINITY, bx1 = -INFINITY, by0 = INFINITY, by1 = -INFINITY;
#pragma unroll
    for (int b = 0; b < kBPL; ++b)
        if (act_body[b]) {
            bx0 = fminf(bx0, px[b]);
            bx1 = fmaxf(bx1, px[b]);
            by0 = fminf(by0, py[b]);
            by1 = fmaxf(by1, py[b]);
        }
    bx0 = warp_min(bx0);
    bx1 = warp_max(bx1);
    by0 = warp_min(by0);
    by1 = warp_max(by1);
    const float gcx = 0.5f * (bx0 + bx1), gcy = 0.5f * (by0 + by1);
    const float ghx = 0.5f * (bx1 - bx0), ghy = 0.5f * (by1 - by0);
    const unsigned below = lanemask_lt();
    // packed operands: the body broadcast to both halves, negated
    float2 nx[kBPL], ny[kBPL], ax2[kBPL], ay2[kBPL];
#pragma unroll
    for (int b = 0; b < kBPL; ++b) {
        nx[b] = make_float2(-px[b], -px[b]);
        ny[b] = make_float2(-py[b], -py[b]);
        ax2[b] = make_float2(0.f, 0.f);
        ay2[b] = make_float2(0.f, 0.f);
    }
    const float2 e2 = make_float2(eps2, eps2);
    ncell = 0;
    npair = 0;
#pragma unroll
    for (int b = 0; b < kBPL; ++b) L.tot[2 * b][lane] = L.tot[2 * b + 1][lane] = make_float2(0.f, 0.f);
    int ccount = 0, bcount = 0, size = 1;
    int flushes = 0;  // warp-uniform: every lane takes part in every flush
    bool shared_top = kShare;
    if (lane == 0) L.stack[0] = root;
    __syncwarp();

    while (size > 0) {
        int k = min(32, size);
        k = min(k, max(1, (kStk - size) / 3));
        const int ref = lane < k ? L.stack[size - k + lane] : 0;
        size -= k;
        __syncwarp();
        int act = 0;  // 1 accept, 2 bodies, 3 open
        int bfirst = 0, bcnt = 0;
        int4 ch = make_int4(INT_MIN, INT_MIN, INT_MIN, INT_MIN);
        float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f);
        float band_d2 = 0.f;
        if (lane < k) {
            if (ref >= 0) {
                c4 = t.cell4[ref];
                const int2 rg = t.range[ref];
                ch = t.child[ref];  // (with the test, not after it: 1,547 -> 1,542 us)
                const bool overlap = !(rg.y < g0 || rg.x > g1);
                const float dx = fmaxf(fabsf(c4.x - gcx) - ghx, 0.f);
                const float dy = fmaxf(fabsf(c4.y - gcy) - ghy, 0.f);
                const float d2 = fmaf(dx, dx, dy * dy);
                band_d2 = d2;
                if (!overlap && c4.w < theta2 * d2) {
                    act = 1;
                } else if (rg.y - rg.x < leaf_size) {
                    act = 2;
                    bfirst = rg.x;
                    bcnt = rg.y - rg.x + 1;
                } else {
                    act = 3;
                }
            } else {
                const int b = ~ref;
                act = 2;
                bfirst = b;
                bcnt = max(0, min(t.leaf_last[b], n - 1) - b + 1);
            }
        }
        if (kShare && shared_top && part > 0 && act != 3) {
            act = 0;
            bcnt = 0;
        }
        // accepted cells
        const unsigned acc_mask = __ballot_sync(kFull, act == 1);
        if (act == 1) {
            const int slot = ccount + __popc(acc_mask & below);
            put_entry(L.cxy, L.cm, slot, c4.x, c4.y, c4.z);
            if (kQuad) {
                const float4 q = t.cellq[ref];
                put_entry(L.qa, L.qb, slot, q.x, q.y, q.z);
            }
        }
        if (kLearned) {
            // band: accepted here but opened by the plain theta_B walk
            const bool in_band = act == 1 && c4.w >= band2 * band_d2;
            const unsigned bm = __ballot_sync(kFull, in_band);
            if (in_band) {
                const int slot = nband + __popc(bm & below);
                if (slot < band_cap) band[slot] = ref;
            }
            nband += __popc(bm);
        }
        ccount += __popc(acc_mask);
        __syncwarp();
        if (ccount >= 32) {
            sum_list<true, kQuad, kZeroSoft, kBPL>(L, 16, one, sl, nx, ny, e2, ax2, ay2,
                                                   ++flushes % kFoldFlushes == 0);
            ncell += 32;
            __syncwarp();
            // pairs 16.. move down; source and destination never overlap
            if (lane < (ccount - 31) / 2) {
                L.cxy[lane] = L.cxy[16 + lane];
                L.cm[lane] = L.cm[16 + lane];
                if (kQuad) {
                    L.qa[lane] = L.qa[16 + lane];
                    L.qb[lane] = L.qb[16 + lane];
                }
            }
            ccount -= 32;
            __syncwarp();
        }
        // opened cells push their children
        const int nch = act == 3 ? (ch.y == INT_MIN ? 1 : ch.z == INT_MIN ? 2 : ch.w == INT_MIN ? 3 : 4)
                                 : 0;
        // One scan for the children (at most 128) and the bodies (at most 2^21;
        // a leaf of more coincident bodies takes a scan of its own): force at 4M
        // 1,577 -> 1,547 us, 1M learned walk 246 -> 240.
        const bool many = __any_sync(kFull, bcnt > 1 << 16);
        int both;
        const int off2 = warp_exclusive_sum(nch + (many ? 0 : bcnt << 8), both);
        const int off = off2 & 255, pushed = both & 255;
        int boff = off2 >> 8, btot = both >> 8;
        if (many) boff = warp_exclusive_sum(bcnt, btot);
        if (size + pushed > kStkAlloc) {  // excluded by the batch rule; stop safely
            if (lane == 0) atomicOr(err, kErrStack);
            break;
        }
        if (act == 3) {
            int* dst = L.stack + size + off;
            dst[0] = ch.x;
            if (nch > 1) dst[1] = ch.y;
            if (nch > 2) dst[2] = ch.z;
            if (nch > 3) dst[3] = ch.w;
        }
        size += pushed;
        // (until then a round takes the whole stack, so size < 4 kShareAt)
        if (kShare && shared_top && size >= kShareAt) {
            shared_top = false;
            __syncwarp();
            const int mine = (size - part + kWarpsPerBlock - 1) / kWarpsPerBlock;
            const int r0 = lane < mine ? L.stack[part + kWarpsPerBlock * lane] : 0;
            __syncwarp();
            if (lane < mine) L.stack[lane] = r0;
            size = mine;
        }
        // the next round's lanes read what other lanes pushed; a round without
        // bodies meets no other barrier on its way there
        __syncwarp();
        // bodies of directly summed cells and leaves, expanded 32 at a time
        for (int base = 0; base < btot; base += 32) {
            const int item = base + lane;
            int owner = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
                const int cand = owner + st;
                const int o = __shfl_sync(kFull, boff, cand);
                if (item >= o) owner = cand;
            }
            const int j = __shfl_sync(kFull, bfirst, owner) + item - __shfl_sync(kFull, boff, owner);
            const int added = min(32, btot - base);
            __syncwarp();
            if (lane < added) {
                const float4 b4 = t.body4[j];
                put_entry(L.bxy, L.bm, bcount + lane, b4.x, b4.y, b4.z);
            }
            bcount += added;
            __syncwarp();
            if (bcount >= 32) {
                sum_list<false, false, kZeroSoft, kBPL>(L, 16, one, sl, nx, ny, e2, ax2, ay2,
                                                        ++flushes % kFoldFlushes == 0);
                npair += 32;
                __syncwarp();
                if (lane < (bcount - 31) / 2) {
                    L.bxy[lane] = L.bxy[16 + lane];
                    L.bm[lane] = L.bm[16 + lane];
                }
                bcount -= 32;
                __syncwarp();
            }
        }
    }
    // odd counts: a padding entry completes the last pair
    if (lane == 0) {
        if (ccount & 1) {
            put_entry(L.cxy, L.cm, ccount, kPadCoord, kPadCoord, 0.f);
            if (kQuad) put_entry(L.qa, L.qb, ccount, 0.f, 0.f, 0.f);
        }
        if (bcount & 1) put_entry(L.bxy, L.bm, bcount, kPadCoord, kPadCoord, 0.f);
    }
    __syncwarp();
    sum_list<true, kQuad, kZeroSoft, kBPL>(L, (ccount + 1) >> 1, one, sl, nx, ny, e2, ax2, ay2, false);
    sum_list<false, false, kZeroSoft, kBPL>(L, (bcount + 1) >> 1, one, sl, nx, ny, e2, ax2, ay2, true);
    ncell += ccount;
    npair += bcount;
#pragma unroll
    for (int b = 0; b < kBPL; ++b) {
        const float2 tx = L.tot[2 * b][lane], ty = L.tot[2 * b + 1][lane];
        ax[b] = tx.x + tx.y;
        ay[b] = ty.x + ty.y;
    }
    // the lanes that share a body
    for (int o = 32 / sl.slots; o < 32; o <<= 1) {
        ax[0] += __shfl_xor_sync(kFull, ax[0], o);
        ay[0] += __shfl_xor_sync(kFull, ay[0], o);
    }
    __syncwarp();
}

// Persistent: each warp takes groups from a global ticket until none is left,
// which balances groups of very different cost.
// Blocks per SM that the walk needs to hide its loads (registers are held to
// what they leave: 64 and 72).
template <bool kQuad, int kBPL>
constexpr int kMinBlocks = kBPL == 4 ? 4 : kQuad && kBPL == 2 ? 7 : 8;

template <bool kQuad, int kBPL, bool kLearned, bool kZeroSoft, bool kShare>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kMinBlocks<kQuad, kBPL>)
force_split(double2* pos, double2* vel, double2* acc_out,
            float2* acc32, int n, Tree t, DeviceScalars* s, Batch bt,
            float eps2, float theta2, int leaf_size, double G_dt, double dt, int kick,
            float band2, unsigned long long* mark, unsigned long long* end) {
    chain_begin();
    mark_start(mark);
    __shared__ WarpLists lists[kWarpsPerBlock];
    const int lane = threadIdx.x & 31;
    __shared__ int block_group;
    const int part = kShare ? threadIdx.x >> 5 : 0;
    WarpLists& L = lists[threadIdx.x >> 5];
    const int ngroups = s->groups;
    unsigned long long cells_total = 0, pairs_total = 0;
    while (true) {
        int g = 0;
        if (kShare) {
            __syncthreads();  // the sums of the last group have been read
            if (threadIdx.x == 0) block_group = (int)atomicAdd(&s->group_ticket, 1u);
            __syncthreads();
            g = block_group;
        } else {
            if (lane == 0) g = (int)atomicAdd(&s->group_ticket, 1u);
            g = __shfl_sync(kFull, g, 0);
        }
        if (g >= ngroups) break;
        const int2 gr = t.groups[g];
        const int g0 = gr.x, g1 = min(gr.y, n - 1);
        // batched universes: walk the group's own universe from its root
        const int root = bt.nuni ? bt.root[bt.uid[g0]] : s->root;
        const double2 fc = frame_center(s, bt, g0);
        const double cx = fc.x, cy = fc.y;
        const int count = g1 - g0 + 1;
        const int width = !kShare || count > 16 ? 32 : count > 8 ? 16 : 8;
        const Slots sl = kShare ? Slots{lane / width, 32 / width} : Slots{0, 1};
        const int place = lane & (width - 1);
        int me[kBPL];
        bool on[kBPL];
        float px[kBPL], py[kBPL], ax[kBPL], ay[kBPL];
#pragma unroll
        for (int b = 0; b < kBPL; ++b) {
            on[b] = 32 * b + place < count;
            me[b] = min(g0 + 32 * b + place, g1);
            const double2 p = pos[me[b]];
            px[b] = (float)(p.x - cx);
            py[b] = (float)(p.y - cy);
        }
        unsigned long long ncell, npair;
        int nband = 0;
        int* band = kLearned ? t.band + (int64_t)kBandPerBody * g0 : nullptr;
        walk_group<kQuad, kBPL, kLearned, kZeroSoft, kShare>(L, t, root, n, g0, g1, count <= 32, sl, px, py, on, eps2, theta2,
                                          leaf_size, ax, ay, ncell, npair, &s->error, band, nband,
                                          kBandPerBody * (g1 - g0 + 1), band2, part);
        if (kShare) {  // the warps' sums, in order
#pragma unroll
            for (int b = 0; b < kBPL; ++b) L.tot[b][lane] = make_float2(ax[b], ay[b]);
            __syncthreads();
#pragma unroll
            for (int b = 0; b < kBPL; ++b)
                for (int w = 1; w < kWarpsPerBlock; ++w) {
                    ax[b] += lists[w].tot[b][lane].x;
                    ay[b] += lists[w].tot[b][lane].y;
                }
        }
        if (kLearned) {
            // the correction kernel adds the learned term, then kicks and drifts
            if (lane == 0) t.band_count[g] = nband;
#pragma unroll
            for (int b = 0; b < kBPL; ++b)
                if (on[b] && sl.slot == 0) acc32[me[b]] = make_float2(ax[b], ay[b]);
        }
#pragma unroll
        for (int b = 0; b < kBPL; ++b) {
            if (kLearned || !on[b] || sl.slot > 0 || part > 0) continue;
            const int i = me[b];
            if (acc_out) acc_out[i] = make_double2((double)ax[b], (double)ay[b]);
            if (kick) {
                double2 v = vel[i];
                v.x += (double)ax[b] * G_dt;
                v.y += (double)ay[b] * G_dt;
                vel[i] = v;
                double2 p = pos[i];  // (read again: not held over the walk)
                p.x += v.x * dt;
                p.y += v.y * dt;
                pos[i] = p;
            }
        }
        // every body of the group summed every entry and skipped itself once
        const unsigned long long bodies = (unsigned long long)(g1 - g0 + 1);
        cells_total += ncell * bodies;
        pairs_total += npair * bodies - (part > 0 ? 0 : bodies);
    }
    if (lane == 0) {
        atomicAdd(&s->cell_terms, cells_total);
        atomicAdd(&s->body_terms, pairs_total);
        if (end) atomicMax(end, global_ns());
    }
}

template <bool kQuad, int kBPL, bool kLearned, bool kZeroSoft, bool kShare>
void launch_split_soft(nb_ctx* c, const BodyBuffers& b, bool kick, bool store_acc, bool chained,
                       float eps2) {
    int& grid = c->split_blocks[(kQuad ? 1 : 0) + (kLearned ? 2 : 0) + (kBPL == 1 ? 4 : 0) +
                                (kBPL == 4 ? 16 : 0) +
                                (kZeroSoft ? 8 : 0) + (kShare ? 32 : 0)];
    if (grid == 0) {
        int blocks = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &blocks, force_split<kQuad, kBPL, kLearned, kZeroSoft, kShare>, kWarpsPerBlock * 32, 0) !=
                    cudaSuccess ||
            blocks < 1) {
            cudaGetLastError();
            blocks = 4;
        }
        grid = c->sm_count * blocks;
    }
    const float theta2 = (float)(c->p.theta * c->p.theta);
    const int leaf = c->p.leaf_size > 0 ? c->p.leaf_size : kDefaultLeaf;
    chain_launch(c->stream, chained, force_split<kQuad, kBPL, kLearned, kZeroSoft, kShare>, grid,
                 32 * kWarpsPerBlock, 0, 1, b.pos, b.vel, store_acc ? c->acc : nullptr, c->acc32,
                 (int)c->n, c->tree, c->scal, c->batch, eps2, theta2, leaf, c->p.G * c->p.timestep,
                 c->p.timestep, kick ? 1 : 0, band_theta(c) * band_theta(c), mark_of(c, 7),
                 kLearned ? nullptr : mark_of(c, kPhases));
}

// The block's four warps walk for one group while all groups fit the GPU at
// once (23 bodies to a group of up to 32: 4,300 of 4,736 resident warps at the
// limit); a group's walk is a chain of some 25 dependent rounds.  Force, us,
// one warp and four: 1,001 bodies 36 and 24, 4,096 45 and 39, 16,384 56 and 47
// (quadrupoles 82 and 69), 32,768 57 and 62.
constexpr int64_t kShareMax = 24576;

// eps2 = 0 takes the variant whose terms skip coincident FP32 points
template <bool kQuad, int kBPL, bool kLearned>
void launch_split_kernel(nb_ctx* c, const BodyBuffers& b, bool kick, bool store_acc,
                         bool chained) {
    // eps2 below the smallest normal float is treated like eps2 = 0
    const float eps2 = (float)c->p.epsilon_squared;
    constexpr bool kCanShare = kBPL == 1 && !kLearned;
    const bool share = kCanShare && bodies_on_148(c) <= kShareMax;
    if (eps2 >= FLT_MIN)
        share ? launch_split_soft<kQuad, kBPL, kLearned, false, kCanShare>(c, b, kick, store_acc, chained, eps2)
              : launch_split_soft<kQuad, kBPL, kLearned, false, false>(c, b, kick, store_acc, chained, eps2);
    else
        share ? launch_split_soft<kQuad, kBPL, kLearned, true, kCanShare>(c, b, kick, store_acc, chained, eps2)
              : launch_split_soft<kQuad, kBPL, kLearned, true, false>(c, b, kick, store_acc, chained, eps2);
}

}  // namespace

int split_group_size(const nb_ctx* c) {
    // learned contexts keep groups of 64 (the correction kernel's layout)
    if (c->p.flags & NB_FLAG_LEARNED) return 32 * kBodiesPerLane;
    return 32 * (c->bpl == 1 ? 1 : c->bpl == 4 ? 4 : kBodiesPerLane);
}

void launch_force_split(nb_ctx* c, const BodyBuffers& b, bool kick, bool store_acc, bool chained) {
    c->launches += 1;
    if (c->p.flags & NB_FLAG_LEARNED) {  // the correction kernel assumes groups of 64
        if (c->p.flags & NB_FLAG_QUADRUPOLE)  // the network corrects the quadrupole walk
            launch_split_kernel<true, kBodiesPerLane, true>(c, b, kick, store_acc, chained);
        else
            launch_split_kernel<false, kBodiesPerLane, true>(c, b, kick, store_acc, chained);
    }
    else if (c->p.flags & NB_FLAG_QUADRUPOLE)
        c->bpl == 1   ? launch_split_kernel<true, 1, false>(c, b, kick, store_acc, chained)
        : c->bpl == 4 ? launch_split_kernel<true, 4, false>(c, b, kick, store_acc, chained)
                      : launch_split_kernel<true, kBodiesPerLane, false>(c, b, kick, store_acc, chained);
    else
        c->bpl == 1   ? launch_split_kernel<false, 1, false>(c, b, kick, store_acc, chained)
        : c->bpl == 4 ? launch_split_kernel<false, 4, false>(c, b, kick, store_acc, chained)
                      : launch_split_kernel<false, kBodiesPerLane, false>(c, b, kick, store_acc, chained);
}

}  // namespace nb
