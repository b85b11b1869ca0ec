// k_allpairs.cu -- FP64 all-pairs accelerations on the GPU: the error oracle
// (nb_allpairs_accelerations) and the NB_MODE_ALLPAIRS step.
//
// a_i = sum_{j != i} m_j d_ij (|d_ij|^2 + eps2)^-3/2, the pair law of the
// reference GPU backend (BarnesHutCuda.cu:427-431) without any tree.  Used to
// state p50/p99 force errors at full size, where a CPU all-pairs sum is too
// slow.  Sources are staged through shared memory in tiles, split over the blocks;
// each thread owns kPer targets.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <string>

#include "nb_internal.cuh"
#include "nbody_b200.h"

namespace {

constexpr int kThreads = 128;
constexpr int kTile = 256;    // sources staged in shared memory at a time

// Pair weight w of a_i += w (p_j - p_i).  kCpuLaw: the law of
// Simulation::force, m / (d (d^2 + eps2)) (Simulation.cpp:74-80, G applied
// with the kick); otherwise Plummer's m (d^2 + eps2)^-3/2.
template <bool kCpuLaw>
__device__ __forceinline__ double pair_weight(double m, double r2, double eps2) {
    return kCpuLaw ? nb::m_over_r_s(m, r2, r2 + eps2)
                   : nb::m_over_r3<false>(m, r2 + eps2);
}
// The same for any r2: zero, subnormal or infinite squares.
template <bool kCpuLaw>
__device__ __forceinline__ double pair_weight_any(double m, double r2, double eps2) {
    if (kCpuLaw) return m / (sqrt(r2) * (r2 + eps2));
    const double inv = 1.0 / sqrt(r2 + eps2);
    return m * inv * inv * inv;
}

// Sums the sources [s0, s1) for the block's targets, kPer per thread: target
// b of a thread is p[b], and self[b] its own source index, which is left out.
// 14 FP64 instructions per pair (15 and a second seed with the CPU law), each
// two issue cycles: the FP64 pipe is the bound, 87% of its cycles active (1 /
// sqrt and its division took some 35 instructions: 65,536 targets of 1,048,576
// bodies with their copies 205 -> 66 ms; a step of 20,011 bodies 0.92 -> 0.37 ms).  Several targets per thread share the loads and
// the loop.  Only a tile that holds one of the warp's own sources tests for
// it; a tile whose sums are not finite (a square that is zero, subnormal or
// infinite, or a term that overflows) is summed again with full-range functions.
template <bool kCpuLaw, int kPer>
__device__ __forceinline__ void sum_sources(const double2* __restrict__ pos,
                                            const double* __restrict__ mass, int64_t s0, int64_t s1,
                                            double eps2, const double2 (&p)[kPer],
                                            const int64_t (&self)[kPer], double (&ax)[kPer],
                                            double (&ay)[kPer]) {
    __shared__ double2 sp[kTile];
    __shared__ double sm[kTile];
    for (int64_t base = s0; base < s1; base += kTile) {
        const int lim = (int)min((int64_t)kTile, s1 - base);
        for (int q = threadIdx.x; q < lim; q += kThreads) {
            sp[q] = pos[base + q];
            sm[q] = mass[base + q];
        }
        __syncthreads();
        double bx[kPer], by[kPer];
        bool own = false, odd = false;
#pragma unroll
        for (int b = 0; b < kPer; ++b) {
            bx[b] = ax[b];
            by[b] = ay[b];
            own |= self[b] >= base && self[b] < base + lim;
        }
        if (!__any_sync(0xffffffffu, own)) {
#pragma unroll 4
            for (int q = 0; q < lim; ++q)
#pragma unroll
                for (int b = 0; b < kPer; ++b) {
                    const double dx = sp[q].x - p[b].x, dy = sp[q].y - p[b].y;
                    const double w = pair_weight<kCpuLaw>(sm[q], fma(dx, dx, dy * dy), eps2);
                    bx[b] = fma(dx, w, bx[b]);
                    by[b] = fma(dy, w, by[b]);
                }
        } else {
            for (int q = 0; q < lim; ++q)
#pragma unroll
                for (int b = 0; b < kPer; ++b) {
                    const double dx = sp[q].x - p[b].x, dy = sp[q].y - p[b].y;
                    const double w = pair_weight<kCpuLaw>(sm[q], fma(dx, dx, dy * dy), eps2);
                    if (base + q != self[b]) {
                        bx[b] = fma(dx, w, bx[b]);
                        by[b] = fma(dy, w, by[b]);
                    }
                }
        }
#pragma unroll
        for (int b = 0; b < kPer; ++b) odd |= !(isfinite(bx[b]) && isfinite(by[b]));
        if (odd) {
            for (int q = 0; q < lim; ++q)
#pragma unroll 1
                for (int b = 0; b < kPer; ++b) {
                    const double dx = sp[q].x - p[b].x, dy = sp[q].y - p[b].y;
                    if (base + q == self[b]) continue;
                    const double w = pair_weight_any<kCpuLaw>(sm[q], fma(dx, dx, dy * dy), eps2);
                    ax[b] += dx * w;
                    ay[b] += dy * w;
                }
        } else {
#pragma unroll
            for (int b = 0; b < kPer; ++b) {
                ax[b] = bx[b];
                ay[b] = by[b];
            }
        }
        __syncthreads();
    }
}

// Block (x, y) sums targets x * kThreads * kPer.. over source chunk y: few
// targets split the sources so that the grid fills the GPU, and the partial
// sums are added in chunk order (deterministic).  targets == nullptr: target
// i is body i.
template <bool kCpuLaw, int kPer>
__global__ void __launch_bounds__(kThreads)
allpairs_partial(const double2* pos, const double* mass, int64_t n,
                 const int64_t* targets, int64_t k, int64_t chunk, double eps2,
                 double2* partial) {
    nb::chain_begin();
    const int64_t first = blockIdx.x * (int64_t)(kThreads * kPer) + threadIdx.x;
    double2 p[kPer];
    int64_t self[kPer];
    double ax[kPer], ay[kPer];
#pragma unroll
    for (int b = 0; b < kPer; ++b) {
        const int64_t i = min(first + b * kThreads, k - 1);
        self[b] = targets ? targets[i] : i;
        p[b] = pos[self[b]];
        ax[b] = ay[b] = 0.0;
    }
    const int64_t s0 = blockIdx.y * chunk, s1 = min(n, s0 + chunk);
    sum_sources<kCpuLaw, kPer>(pos, mass, s0, s1, eps2, p, self, ax, ay);
#pragma unroll
    for (int b = 0; b < kPer; ++b) {
        const int64_t i = first + b * kThreads;
        if (i < k) partial[blockIdx.y * k + i] = make_double2(ax[b], ay[b]);
    }
}

// Target i's partial sums added in chunk order (loads of eight in flight).
__device__ __forceinline__ double2 fold_partial(const double2* __restrict__ partial, int chunks,
                                                int64_t k, int64_t i) {
    double ax = 0.0, ay = 0.0;
#pragma unroll 8
    for (int c = 0; c < chunks; ++c) {
        const double2 a = partial[c * k + i];
        ax += a.x;
        ay += a.y;
    }
    return make_double2(ax, ay);
}

__global__ void allpairs_fold(const double2* __restrict__ partial, int chunks, int64_t k,
                              double2* __restrict__ acc) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < k) acc[i] = fold_partial(partial, chunks, k, i);
}

// NB_MODE_ALLPAIRS, stage 1 (AllPairs.cpp:31-35): b = a with x += v dt (or a
// plain copy when only accelerations are wanted).
__global__ void allpairs_drift(nb::BodyBuffers a, nb::BodyBuffers b, int64_t n, double dt,
                               nb::DeviceScalars* s, unsigned long long* mark) {
    nb::chain_begin();
    nb::mark_start(mark);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->cell_terms = 0;
        s->body_terms = 0;
        s->stack_hw = 0;
    }
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2 p = a.pos[i], v = a.vel[i];
    // x + v dt rounded twice, as the reference's `pos += vel * timestep`
    b.pos[i] = make_double2(__dadd_rn(p.x, __dmul_rn(v.x, dt)), __dadd_rn(p.y, __dmul_rn(v.y, dt)));
    b.vel[i] = v;
    b.mass[i] = a.mass[i];
    b.orig[i] = a.orig[i];
}

// Stage 2 (AllPairs.cpp:38-49): every body sums all others (allpairs_partial;
// each pair is evaluated from both sides: twice the reference's pair
// evaluations, no atomics), then the kick.
__global__ void allpairs_kick(const double2* partial, int chunks, int64_t n,
                              double2* vel, double2* acc_out,
                              double G_dt, int kick, unsigned long long* body_terms,
                              unsigned long long* end) {
    nb::chain_begin();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2 a = fold_partial(partial, chunks, n, i);
    if (acc_out) acc_out[i] = a;
    if (kick) {
        double2 v = vel[i];
        v.x += a.x * G_dt;
        v.y += a.y * G_dt;
        vel[i] = v;
    }
    if (threadIdx.x == 0)
        atomicAdd(body_terms, (unsigned long long)min((int64_t)blockDim.x, n - i) * (n - 1));
    nb::mark_end(end);
}

// Two targets per thread share each source's load; below this many targets
// one per thread fills the GPU better.
constexpr int64_t kTwoPerThread = 16384;

inline int64_t target_blocks(int64_t k) {
    const int64_t per = kThreads * (k >= kTwoPerThread ? 2 : 1);
    return (k + per - 1) / per;
}

// Source chunks for k targets and n sources: four waves of eight blocks per
// SM, so that the last wave costs little (and the partial sums, 16 bytes per
// target and chunk, stay below 20 MB), with chunks of at least 32 sources.
inline int source_chunks(int64_t k, int64_t n, int sm_count) {
    const int64_t want = (int64_t)sm_count * 8 * 4 / target_blocks(k);
    return (int)std::max<int64_t>(1, std::min<int64_t>({want, n / 32, 256}));
}

template <bool kCpuLaw>
void launch_partial(const double2* pos, const double* mass, int64_t n, const int64_t* targets,
                    int64_t k, int chunks, double eps2, double2* partial, cudaStream_t st,
                    bool chained) {
    const dim3 grid((unsigned)target_blocks(k), (unsigned)chunks);
    const int64_t chunk = (n + chunks - 1) / chunks;
    nb::chain_launch(st, chained,
                     k >= kTwoPerThread ? allpairs_partial<kCpuLaw, 2> : allpairs_partial<kCpuLaw, 1>,
                     grid, kThreads, 0, 1, pos, mass, n, targets, k, chunk, eps2, partial);
}

}  // namespace

int nb::allpairs_chunks(int64_t n, int sm_count) { return source_chunks(n, n, sm_count); }

void nb::launch_allpairs_step(nb_ctx* c, const BodyBuffers& a, const BodyBuffers& b, bool integrate,
                              bool store_acc) {
    const unsigned blocks = (unsigned)((c->n + kThreads - 1) / kThreads);
    const int chunks = allpairs_chunks(c->n, c->sm_count);
    c->launches += 3;
    chain_launch(c->stream, false, allpairs_drift, blocks, kThreads, 0, 1, a, b, c->n,
                 integrate ? c->p.timestep : 0.0, c->scal, mark_of(c, 7));
    if (c->p.flags & NB_FLAG_CPU_LAW)
        launch_partial<true>(b.pos, b.mass, c->n, nullptr, c->n, chunks, c->p.epsilon_squared,
                             c->ap_partial, c->stream, true);
    else
        launch_partial<false>(b.pos, b.mass, c->n, nullptr, c->n, chunks, c->p.epsilon_squared,
                              c->ap_partial, c->stream, true);
    chain_launch(c->stream, true, allpairs_kick, blocks, kThreads, 0, 1, c->ap_partial, chunks, c->n,
                 b.vel, store_acc ? c->acc : nullptr, c->p.G * c->p.timestep, integrate ? 1 : 0,
                 &c->scal->body_terms, mark_of(c, kPhases));
}

extern "C" int nb_allpairs_accelerations(int32_t device, uint64_t n, const double* mass,
                                         const double* pos_xy, uint64_t k, const int64_t* targets,
                                         double epsilon_squared, double* acc_xy) {
    if (!mass || !pos_xy || !targets || !acc_xy || n == 0 || k == 0) return NB_ERR_INVALID;
    if (!std::isfinite(epsilon_squared) || epsilon_squared < 0.0) return NB_ERR_INVALID;
    for (uint64_t i = 0; i < k; ++i)
        if (targets[i] < 0 || (uint64_t)targets[i] >= n) return NB_ERR_INVALID;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return NB_ERR_NOTFOUND;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    double2 *dpos = nullptr, *dacc = nullptr, *dpart = nullptr;
    double* dmass = nullptr;
    int64_t* dtgt = nullptr;
    cudaStream_t st = nullptr;
    int rc = NB_OK, sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int chunks = source_chunks((int64_t)k, (int64_t)n, sms > 0 ? sms : 1);
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&dpos, n * sizeof(double2)) != cudaSuccess ||
        cudaMalloc(&dmass, n * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&dtgt, k * sizeof(int64_t)) != cudaSuccess ||
        cudaMalloc(&dacc, k * sizeof(double2)) != cudaSuccess ||
        (chunks > 1 && cudaMalloc(&dpart, k * chunks * sizeof(double2)) != cudaSuccess)) {
        rc = NB_ERR_NOMEM;
    }
    if (rc == NB_OK) {
        cudaMemcpyAsync(dpos, pos_xy, n * sizeof(double2), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dmass, mass, n * sizeof(double), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dtgt, targets, k * sizeof(int64_t), cudaMemcpyHostToDevice, st);
        launch_partial<false>(dpos, dmass, (int64_t)n, dtgt, (int64_t)k, chunks, epsilon_squared,
                              chunks > 1 ? dpart : dacc, st, false);
        if (chunks > 1)
            allpairs_fold<<<(unsigned)((k + kThreads - 1) / kThreads), kThreads, 0, st>>>(
                dpart, chunks, (int64_t)k, dacc);
        cudaMemcpyAsync(acc_xy, dacc, k * sizeof(double2), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
            rc = NB_ERR_CUDA;
    }
    cudaFree(dpos);
    cudaFree(dmass);
    cudaFree(dtgt);
    cudaFree(dacc);
    cudaFree(dpart);
    if (st) cudaStreamDestroy(st);
    cudaSetDevice(prev);
    return rc;
}
