// k_force64.cu -- FP64 parity traversal, kick, drift and the original-order
// scatter.
//
// The traversal keeps the reference's semantics (BarnesHutCuda.cu:382-486):
// the per-body opening test width^2 < theta^2 d^2 against the cell's centre of
// mass, the Plummer pair law a += d m (d^2 + eps^2)^-3/2, no opening test for
// a multi-body leaf that does not hold the target, and the kick v += a G dt.
// On the compressed tree a cell is tested at its own (deepest-chain) level,
// which decides exactly as the reference's chain does; a multi-body leaf that
// holds the target is first tested at level 29 when the reference reaches it
// through a chain of single-child cells, because the reference may accept
// such a chain (and so the target's own mass) when theta > 1/sqrt(2).
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nb_internal.cuh"

namespace nb {
namespace {

constexpr int kWarpsPerBlock = 4;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kStk = 256;             // stack bound kept by the batch size rule
constexpr int kStkAlloc = kStk + 96;  // + one depth-first descent (<= 3 x 30 + 1)
constexpr int kListCap = 64;          // flushed 32 entries at a time

// Shared memory of one warp.
struct Walk64 {
    int2 stack[kStkAlloc];       // {cell or ~leaf, bodies of the group that reached it}
    double2 fxy[kListCap];       // interaction list: position
    double fm[kListCap];         //   and mass
    double2 pxy[kListCap + 1];   // list of entries that act on some bodies only,
    double pm[kListCap + 1];     //   ended by an entry of no mass
    unsigned mask[kListCap];     // the bodies that the entries act on
    double2 nxy[32];             // cells that need the per-body test: COM
    double nw[32];               //   and squared width
};

// The reference's squared distance (nvcc contracts CU:461 to this fma).
// Rounding is monotone, so it never decreases when |dx| or |dy| grows.
__device__ __forceinline__ double dist2(double dx, double dy) {
    return __fma_rn(dx, dx, __dmul_rn(dy, dy));
}

__device__ __forceinline__ void plummer(double dx, double dy, double m, double eps2, double& ax,
                                        double& ay) {
    const double d2 = dist2(dx, dy) + eps2;
    double a = m_over_r3<true>(m, d2);
    if (!isfinite(a)) a = m_over_r3_any(m, d2);
    ax += dx * a;
    ay += dy * a;
}

// One warp per group of kG sorted bodies walks the union of their trees.  The
// stack holds nodes with the mask of the bodies that reached them; each round
// pops up to 32 nodes, one per lane.  A cell is first compared with the
// group's bounding box: dx and dy to the box's nearest and farthest sides
// bound every body's |dx| and |dy| after rounding too (rounding is monotone),
// so "accepted at the nearest" and "opened at the farthest" are exactly what
// each body's own test says.  Cells in between are tested by the bodies, lane
// = body.  Every body therefore interacts with exactly the cells and bodies
// of its own depth-first walk (CU:382-486), only the order of the sum differs.
// Accepted nodes go to a shared-memory list, which the warp sums 32 entries at
// a time: lane = (list slot, body), 32 / kG slots side by side.
//
// At 1M bodies issue is at 70% and the FP64 pipe at 50% of its cycles (14
// instructions per body and list entry, each two issue cycles, and the opening
// tests): no unit is full, fixed latencies and turns at issue take the rest.  One
// thread per body and one node at a time kept the pipe at 16% and 18 of 32 lanes
// active: scattered loads behind every step of a serial walk.
// kTerms (nb_debug_interactions): per-body interaction counts and the depth
// a depth-first walk's stack would reach.  A node's pending count (siblings
// waiting at and above it) is a property of its path, so each node carries it.
template <int kG, bool kTerms>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 7)
force_fp64(const double2* pos, const double* mass, double2* vel,
           double2* acc_out, int n, Tree t, DeviceScalars* s, double eps2,
           double theta_sq, double G_dt, int kick, uint2* terms_out,
           unsigned long long* mark) {
    chain_begin();
    mark_start(mark);
    static_assert(kG >= 1 && kG <= 32 && (kG & (kG - 1)) == 0, "a power of two of bodies per warp");
    constexpr int kSlots = 32 / kG;
    // At kG = 32 more than half of a group's entries act on some 9 bodies each:
    // these go to a list of their own, summed body by body.  Small groups, whose
    // entries mostly act on all bodies, keep one list and leave bodies out (kG =
    // 4 at 16,384 bodies 55 us, with two lists 61; kG = 32 at 1,048,576 bodies
    // 1.18 ms with one list, 1.06 with two).
    constexpr bool kColumns = kG >= 16;
    constexpr bool kMasked = kG > 1 && !kColumns;
    constexpr unsigned kGroupMask = kG == 32 ? kFull : (1u << kG) - 1u;
    __shared__ Walk64 walks[kWarpsPerBlock];
    __shared__ double wsq[kMaxLevel + 1];
    __shared__ uint8_t pends[kTerms ? kWarpsPerBlock : 1][kTerms ? kStkAlloc : 1];
    if (threadIdx.x <= kMaxLevel) wsq[threadIdx.x] = s->wsq[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g0l = ((int64_t)blockIdx.x * kWarpsPerBlock + warp) * kG;
    if (g0l >= n) return;
    Walk64& L = walks[warp];
    uint8_t* pend = pends[kTerms ? warp : 0];
    const int g0 = (int)g0l, count = min(kG, n - g0);
    const int body = lane & (kG - 1), slot = lane / kG;
    const bool on = body < count;
    const double2 me = pos[g0 + min(body, count - 1)];
    // the group's box (lanes past the end hold the last body again)
    double bx0 = me.x, bx1 = me.x, by0 = me.y, by1 = me.y;
#pragma unroll
    for (int o = 1; o < kG; o <<= 1) {
        bx0 = fmin(bx0, __shfl_xor_sync(kFull, bx0, o));
        bx1 = fmax(bx1, __shfl_xor_sync(kFull, bx1, o));
        by0 = fmin(by0, __shfl_xor_sync(kFull, by0, o));
        by1 = fmax(by1, __shfl_xor_sync(kFull, by1, o));
    }
    const int cells = s->cells;
    const unsigned below = lanemask_lt();
    double ax = 0.0, ay = 0.0;
    unsigned long long ncell = 0, npair = 0;  // summed over the group, split over the lanes
    unsigned my_cells = 0, my_pairs = 0;      // kTerms: this lane's body and slots
    unsigned full_cells = 0, full_pairs = 0;  // kTerms: entries of the full list
    unsigned long long pkinds = 0;            // kTerms: single bodies in the partial list
    int deepest = 1, size = 1, fcount = 0, pcount = 0;
    const unsigned whole = count == 32 ? kFull : (1u << count) - 1u;
    if (lane == 0) {
        L.stack[0] = make_int2(s->root, (int)whole);
        L.pxy[kListCap] = make_double2(1e15, 1e15);
        L.pm[kListCap] = 0.0;
        if (kTerms) pend[0] = 0;
    }
    __syncwarp();

    // Both lists below take the first cnt <= 32 entries.  A term whose d2 is
    // zero, subnormal or infinite, or that overflows, comes out infinite or NaN:
    // such a batch (almost never) is summed again, these terms with the
    // full-range 1/sqrt.
    auto sum_full = [&](int cnt) {
        const double ax0 = ax, ay0 = ay;
#pragma unroll 4
        for (int k = slot; k < cnt; k += kSlots) {
            const double2 p = L.fxy[k];
            const double dx = p.x - me.x, dy = p.y - me.y;
            const double a = m_over_r3<true>(L.fm[k], dist2(dx, dy) + eps2);
            if (!kMasked || ((L.mask[k] >> body) & 1u)) {
                ax = fma(dx, a, ax);
                ay = fma(dy, a, ay);
            }
        }
        if (__any_sync(kFull, !(isfinite(ax) && isfinite(ay)))) {
            ax = ax0;
            ay = ay0;
            for (int k = slot; k < cnt; k += kSlots) {
                const double2 p = L.fxy[k];
                if (!kMasked || ((L.mask[k] >> body) & 1u))
                    plummer(p.x - me.x, p.y - me.y, L.fm[k], eps2, ax, ay);
            }
        }
        __syncwarp();
    };
    // Each body takes its own entries: its column of the 32 x 32 mask matrix.
    auto sum_part = [&](int cnt, unsigned kinds) {
        unsigned mine = warp_transpose_bits(lane < cnt ? L.mask[lane] : 0u);
        if (kG < 32) {
            mine = __shfl_sync(kFull, mine, body);
            unsigned of_slot = 0;
#pragma unroll
            for (int k = 0; k < 32; k += kSlots) of_slot |= 1u << k;
            mine &= of_slot << slot;
        }
        if (kTerms) {
            my_pairs += __popc(mine & kinds);
            my_cells += __popc(mine & ~kinds);
        }
        const double ax0 = ax, ay0 = ay;
        const unsigned all = mine;
        const int most = __reduce_max_sync(kFull, __popc(mine));
#pragma unroll 2
        for (int q = 0; q < most; ++q) {
            const int k = mine ? __ffs(mine) - 1 : kListCap;
            mine &= mine - 1;
            const double2 p = L.pxy[k];
            const double dx = p.x - me.x, dy = p.y - me.y;
            const double a = m_over_r3<true>(L.pm[k], dist2(dx, dy) + eps2);
            ax = fma(dx, a, ax);
            ay = fma(dy, a, ay);
        }
        if (__any_sync(kFull, !(isfinite(ax) && isfinite(ay)))) {
            ax = ax0;
            ay = ay0;
            for (unsigned rest = all; rest; rest &= rest - 1) {
                const int k = __ffs(rest) - 1;
                const double2 p = L.pxy[k];
                plummer(p.x - me.x, p.y - me.y, L.pm[k], eps2, ax, ay);
            }
        }
        __syncwarp();
    };

    while (size > 0) {
        int k = min(32, size);
        k = min(k, max(1, (kStk - size) / 3));
        int2 e = make_int2(0, 0);
        int pd = 0;
        if (lane < k) {
            e = L.stack[size - k + lane];
            if (kTerms) pd = pend[size - k + lane];
        }
        size -= k;
        __syncwarp();
        const unsigned mask = (unsigned)e.y;  // empty for lanes without a node
        unsigned accept = 0, open = 0, inside = 0;
        bool single = false;
        bool test = false;
        int first = 0, last = 0;
        double m = 0.0, w = 0.0;
        double2 c = make_double2(0.0, 0.0);
        int4 ch = make_int4(INT_MIN, INT_MIN, INT_MIN, INT_MIN);
        if (mask && e.x >= 0) {
            int lv = -1;
            // one round of loads, none waiting for the level (1,001 bodies 21.5 ->
            // 18.7 us, 300k 384 -> 375, 1M 1,044 -> 1,037)
            if (e.x < cells) {
                lv = t.level[e.x];
                m = t.mass[e.x];
                c = t.com[e.x];
                ch = t.child[e.x];
            }
            if (lv < 0 || lv >= kMaxLevel) {
                atomicOr(&s->error, kErrTree);
            } else {
                w = wsq[lv];
                // nearest and farthest side of the box
                const double x0 = bx0 - c.x, x1 = c.x - bx1, y0 = by0 - c.y, y1 = c.y - by1;
                const double xn = x0 > x1 ? x0 : x1, yn = y0 > y1 ? y0 : y1;
                // (an undefined centre keeps its NaN, which fails both tests below)
                const double near2 = dist2(xn < 0.0 ? 0.0 : xn, yn < 0.0 ? 0.0 : yn);
                if (w < theta_sq * near2) {
                    accept = mask;
                } else if (kG == 1) {
                    open = mask;  // the box is the body: the near test was its own
                } else {
                    const double far2 = dist2(x0 > x1 ? x1 : x0, y0 > y1 ? y1 : y0);
                    if (w < theta_sq * far2) test = true; else open = mask;
                }
            }
        } else if (mask) {
            first = ~e.x;
            last = -1;
            if (first < n) {
                last = t.leaf_last[first];
                c = pos[first];  // of a single body, CU:424-433
                m = mass[first];
            }
            if (last < first || last >= n) {
                atomicOr(&s->error, kErrTree);
            } else {
                // the group's bodies that lie in the leaf
                const int a = max(first - g0, 0), b = min(last - g0, kG - 1);
                inside = b >= a ? (kFull >> (31 - (b - a))) << a : 0u;
                accept = mask & ~inside;
                inside &= mask;
                if (first == last) {
                    single = true;
                    inside = 0;
                } else {  // CU:434-442; the bodies inside: below
                    c = t.bucket_com[first];
                    m = t.bucket_mass[first];
                }
            }
        }
        if (kG > 1) {
            const unsigned tests = __ballot_sync(kFull, test);
            if (tests) {
                const int rank = __popc(tests & below), ntest = __popc(tests);
                if (test) {
                    L.nxy[rank] = c;
                    L.nw[rank] = w;
                }
                __syncwarp();
#pragma unroll 2
                for (int q = 0; q < ntest; q += kSlots) {
                    const int j = q + slot;
                    bool pass = false;
                    if (j < ntest) {
                        const double2 p = L.nxy[j];
                        pass = L.nw[j] < theta_sq * dist2(p.x - me.x, p.y - me.y);
                    }
                    const unsigned bal = __ballot_sync(kFull, pass);
                    if (test && rank >= q && rank < q + kSlots) {
                        const unsigned ok = (bal >> ((rank - q) * kG)) & kGroupMask;
                        accept = mask & ok;
                        open = mask & ~ok;
                    }
                }
                __syncwarp();
            }
        }
        if (accept) {
            if (single) npair += __popc(accept); else ncell += __popc(accept);
        }
        const bool to_part = kColumns && accept && accept != whole;
        const bool to_full = accept && !to_part;
        const unsigned full_lanes = __ballot_sync(kFull, to_full);
        const unsigned part_lanes = kColumns ? __ballot_sync(kFull, to_part) : 0u;
        if (to_full) {
            const int at = fcount + __popc(full_lanes & below);
            L.fxy[at] = c;
            L.fm[at] = m;
            if (kMasked) L.mask[at] = accept;
        }
        if (to_part) {
            const int at = pcount + __popc(part_lanes & below);
            L.pxy[at] = c;
            L.pm[at] = m;
            L.mask[at] = accept;
        }
        if (kTerms) {
            const unsigned f1 = __ballot_sync(kFull, to_full && single);
            full_pairs += __popc(f1);
            full_cells += __popc(full_lanes & ~f1);
            // the partial list's kinds, entry by entry
            for (unsigned rest = part_lanes, at = pcount; rest; rest &= rest - 1, ++at) {
                const unsigned long long bit =
                    __shfl_sync(kFull, (int)single, __ffs(rest) - 1) ? 1ull << at : 0ull;
                pkinds |= bit;
            }
        }
        fcount += __popc(full_lanes);
        pcount += __popc(part_lanes);
        __syncwarp();
        if (fcount >= 32) {
            sum_full(32);
            fcount -= 32;
            if (lane < fcount) {  // source and destination never overlap
                L.fxy[lane] = L.fxy[32 + lane];
                L.fm[lane] = L.fm[32 + lane];
                if (kMasked) L.mask[lane] = L.mask[32 + lane];
            }
            __syncwarp();
        }
        if (kColumns && pcount >= 32) {
            sum_part(32, (unsigned)pkinds);
            pkinds >>= 32;
            pcount -= 32;
            if (lane < pcount) {
                L.pxy[lane] = L.pxy[32 + lane];
                L.pm[lane] = L.pm[32 + lane];
                L.mask[lane] = L.mask[32 + lane];
            }
            __syncwarp();
        }
        // bodies that share a multi-body leaf with the target (CU:443-457), the
        // leaf's bodies spread over the slots
        for (unsigned rest = __ballot_sync(kFull, inside != 0); rest; rest &= rest - 1) {
            const int q = __ffs(rest) - 1;
            const int b = __shfl_sync(kFull, first, q), en = __shfl_sync(kFull, last, q);
            const unsigned who = __shfl_sync(kFull, inside, q);
            if ((who >> body) & 1u) {
                const double2 bc = t.bucket_com[b];
                const double dx = bc.x - me.x, dy = bc.y - me.y;
                if (t.leaf_plevel[b] < kMaxLevel - 1 &&
                    wsq[kMaxLevel - 1] < theta_sq * dist2(dx, dy)) {
                    if (slot == 0) {
                        plummer(dx, dy, t.bucket_mass[b], eps2, ax, ay);
                        ++ncell;
                        ++my_cells;
                    }
                } else {
                    for (int j = b + slot; j <= en; j += kSlots) {
                        if (j == g0 + body) continue;
                        const double2 p = pos[j];
                        plummer(p.x - me.x, p.y - me.y, mass[j], eps2, ax, ay);
                        ++npair;
                        ++my_pairs;
                    }
                }
            }
            __syncwarp();
        }
        // opened cells push their children with the bodies that opened them
        const int nch =
            !open ? 0 : ch.y == INT_MIN ? 1 : ch.z == INT_MIN ? 2 : ch.w == INT_MIN ? 3 : 4;
        int inc = nch;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, inc, o);
            if (lane >= o) inc += v;
        }
        const int pushed = __shfl_sync(kFull, inc, 31);
        if (size + pushed > kStkAlloc) {  // excluded by the batch rule; stop safely
            if (lane == 0) atomicOr(&s->error, kErrStack);
            break;
        }
        if (open) {
            const int at = size + inc - nch;
            const int refs[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nch) {
                    L.stack[at + q] = make_int2(refs[q], (int)open);
                    if (kTerms) pend[at + q] = (uint8_t)(pd + nch - 1 - q);
                }
            if (kTerms) deepest = max(deepest, pd + nch);
        }
        size += pushed;
        __syncwarp();
    }
    sum_full(fcount);
    if (kColumns) sum_part(pcount, (unsigned)pkinds);
    if (kTerms && slot == 0) {
        my_cells += full_cells;
        my_pairs += full_pairs;
    }
#pragma unroll
    for (int o = kG; o < 32; o <<= 1) {
        ax += __shfl_xor_sync(kFull, ax, o);
        ay += __shfl_xor_sync(kFull, ay, o);
        if (kTerms) {
            my_cells += __shfl_xor_sync(kFull, my_cells, o);
            my_pairs += __shfl_xor_sync(kFull, my_pairs, o);
        }
    }
    if (slot == 0 && on) {
        const int i = g0 + body;
        if (acc_out) acc_out[i] = make_double2(ax, ay);
        if (kTerms && terms_out) terms_out[i] = make_uint2(my_cells, my_pairs);
        if (kick) {
            double2 v = vel[i];
            v.x += ax * G_dt;
            v.y += ay * G_dt;
            vel[i] = v;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        ncell += __shfl_xor_sync(kFull, ncell, o);
        npair += __shfl_xor_sync(kFull, npair, o);
        if (kTerms) deepest = max(deepest, __shfl_xor_sync(kFull, deepest, o));
    }
    if (lane == 0) {
        atomicAdd(&s->cell_terms, ncell);
        atomicAdd(&s->body_terms, npair);
        if (kTerms) atomicMax(&s->stack_hw, deepest);
    }
}

template <int kG, bool kTerms>
void launch_walk64(nb_ctx* c, const BodyBuffers& b, bool kick, bool store_acc) {
    const int64_t groups = (c->n + kG - 1) / kG;
    chain_launch(c->stream, true, force_fp64<kG, kTerms>,
                 (unsigned)((groups + kWarpsPerBlock - 1) / kWarpsPerBlock), kWarpsPerBlock * 32, 0, 1,
                 b.pos, b.mass, b.vel, store_acc ? c->acc : nullptr, (int)c->n, c->tree, c->scal,
                 c->p.epsilon_squared, c->p.theta * c->p.theta, c->p.G * c->p.timestep, kick ? 1 : 0,
                 kTerms ? c->dbg_terms : nullptr, mark_of(c, 7));
}

// Drift, CU:489-495.
__global__ void drift_kernel(double2* pos, const double2* vel, int64_t n,
                             double dt, unsigned long long* mark, unsigned long long* end) {
    chain_begin();
    mark_start(mark);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) {
        double2 p = pos[i];
        const double2 v = vel[i];
        p.x += v.x * dt;
        p.y += v.y * dt;
        pos[i] = p;
    }
    mark_end(end);
}

// CU:498-506, plus the optional accelerations.
__global__ void scatter_kernel(const double2* __restrict__ pos, const double2* __restrict__ vel,
                               const int32_t* __restrict__ orig, int64_t n, double2* out_pos,
                               double2* out_vel, const double2* __restrict__ acc,
                               double2* out_acc) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t o = orig[i];
    if (out_pos) out_pos[o] = pos[i];
    if (out_vel) out_vel[o] = vel[i];
    if (out_acc) out_acc[o] = acc[i];
}

// Uploaded bodies: orig = identity, and the checks nb_upload promises
// (finite positions and velocities, positive finite masses) done on the
// device: bit 0 of *bad for a non-finite value, bit 1 for a mass <= 0.
__global__ void upload_kernel(int32_t* __restrict__ orig, const double* __restrict__ mass,
                              const double2* __restrict__ pos, const double2* __restrict__ vel,
                              int64_t n, unsigned* __restrict__ bad) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (orig) orig[i] = (int32_t)i;
    const double m = mass[i];
    const double2 p = pos[i], v = vel[i];
    unsigned f = 0;
    if (!(isfinite(m) && isfinite(p.x) && isfinite(p.y) && isfinite(v.x) && isfinite(v.y))) f |= 1u;
    if (!(m > 0.0)) f |= 2u;
    if (__any_sync(__activemask(), f != 0) && f) atomicOr(bad, f);
}

// Moves checked staged bodies into the state in original order.  After a
// rejected check the state keeps its bodies: when they live in another
// buffer (keep != dst) they are copied over, since the next step reads dst.
__global__ void upload_commit(const double* __restrict__ sm, const double2* __restrict__ sp,
                              const double2* __restrict__ sv, BodyBuffers keep, BodyBuffers dst,
                              int64_t n, const unsigned* __restrict__ bad,
                              unsigned* __restrict__ err) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (*bad) {
        if (i == 0) atomicOr(err, kErrUpload);
        if (keep.mass == dst.mass) return;
        dst.orig[i] = keep.orig[i];
        dst.mass[i] = keep.mass[i];
        dst.pos[i] = keep.pos[i];
        dst.vel[i] = keep.vel[i];
        return;
    }
    dst.orig[i] = (int32_t)i;
    dst.mass[i] = sm[i];
    dst.pos[i] = sp[i];
    dst.vel[i] = sv[i];
}

__global__ void identity_kernel(int32_t* orig, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) orig[i] = (int32_t)i;
}

inline unsigned blocks_for(int64_t n, int threads) {
    return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

void launch_force_fp64(nb_ctx* c, const BodyBuffers& b, bool kick, bool store_acc) {
    c->launches += 1;
    if (c->want_terms) return launch_walk64<32, true>(c, b, kick, store_acc);
    // A warp's walk is a chain of dependent loads, which a smaller group shortens,
    // while a larger one shares each node among more bodies: few enough bodies per
    // warp that the walk is between one and two waves of the resident warps (4,144
    // = 148 SMs x 28), two just below each switch.  Force, us, at kG = 1 / 2 / 4 / 8
    // / 16 / 32, Plummer disc: 6,000 bodies 53 / 36 / 36 / 45 / 64 / 80; 8,191 61 /
    // 42 / 41 / 48 / 69 / 82; 16,383 128 / 83 / 54 / 55 / 76 / 88; 32,767 293 / 174 /
    // 104 / 74 / 89 / 101; 65,535 681 / 388 / 226 / 147 / 120 / 127; 131,071 1529 /
    // 840 / 474 / 292 / 218 / 186; 200,003 2456 / 1330 / 737 / 446 / 317 / 269.  The
    // next size would be the quicker one from about two thirds of the way to its
    // switch on (at 8,191 41 instead of 61, at 32,767 74 instead of 104).  1,048,576
    // bodies take 1,037 at kG = 32, 3,596 with one thread per body.
    const int64_t per_warp = bodies_on_148(c) / 4096;
    if (per_warp < 2) return launch_walk64<1, false>(c, b, kick, store_acc);
    if (per_warp < 4) return launch_walk64<2, false>(c, b, kick, store_acc);
    if (per_warp < 8) return launch_walk64<4, false>(c, b, kick, store_acc);
    if (per_warp < 16) return launch_walk64<8, false>(c, b, kick, store_acc);
    if (per_warp < 32) return launch_walk64<16, false>(c, b, kick, store_acc);
    launch_walk64<32, false>(c, b, kick, store_acc);
}

void launch_drift(nb_ctx* c, const BodyBuffers& b) {
    c->launches += 1;
    chain_launch(c->stream, true, drift_kernel, blocks_for(c->n, 256), 256, 0, 1, b.pos, b.vel, c->n,
                 c->p.timestep, mark_of(c, 8), mark_of(c, kPhases));
}

void launch_scatter(nb_ctx* c, const BodyBuffers& b, double2* out_pos, double2* out_vel,
                    const double2* acc, double2* out_acc) {
    c->launches += 1;
    scatter_kernel<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(b.pos, b.vel, b.orig, c->n, out_pos,
                                                                 out_vel, acc, out_acc);
}

void launch_identity(nb_ctx* c, int32_t* orig) {
    c->launches += 1;
    identity_kernel<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(orig, c->n);
}

void launch_upload_commit(nb_ctx* c, const double* m, const double2* p, const double2* v,
                          const BodyBuffers& keep, const BodyBuffers& dst, unsigned* bad) {
    c->launches += 2;
    cudaMemsetAsync(bad, 0, sizeof(unsigned), c->stream);
    upload_kernel<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(nullptr, m, p, v, c->n, bad);
    upload_commit<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(m, p, v, keep, dst, c->n, bad,
                                                                 &c->scal->error);
}

void launch_upload_check(nb_ctx* c, const BodyBuffers& b, unsigned* bad) {
    c->launches += 1;
    upload_kernel<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(b.orig, b.mass, b.pos, b.vel, c->n,
                                                                 bad);
}

}  // namespace nb
