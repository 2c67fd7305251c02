// apgd_common.cuh -- pieces shared by the persistent APGD kernels: bounded grid barrier,
// fixed-order block reductions, vector loads and the friction-cone projection.
#pragma once
#include <math.h>

#include "kernels.cuh"

namespace scopi_gpu {
namespace apgdc {

constexpr int kThreadsA = 256;
constexpr unsigned long long kBarrierTimeoutNs = 20ull * 1000ull * 1000ull * 1000ull;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barrier words of a persistent launch (the host writes all four before the launch):
// bar[0] = arrivals, bar[1] = generation, bar[2] = error flag, bar[3] = wait limit in
// microseconds (0: kBarrierTimeoutNs).
__device__ __forceinline__ unsigned long long barrier_limit_ns(const unsigned int* bar) {
    const unsigned int us = *(volatile const unsigned int*)(bar + 3);
    return us ? (unsigned long long)us * 1000ull : kBarrierTimeoutNs;
}

// Grid-wide barrier for a cooperative launch.  A block that waits longer than the limit
// sets the error flag and returns false; every waiting block sees the flag and returns
// false too, so the kernel ends with an error status instead of hanging.  withhold: this
// block does not count itself (used once, to test that path: the barrier then never
// completes and every block gives up after the limit).
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int nblocks, bool withhold = false) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned int* vgen = bar + 1;
        volatile unsigned int* verr = bar + 2;
        const unsigned int gen = *vgen;
        __threadfence();
        const unsigned int arrived = withhold ? 0u : atomicAdd(bar, 1u);
        if (!withhold && arrived == nblocks - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            const unsigned long long t0 = global_ns(), limit = barrier_limit_ns(bar);
            unsigned int it = 0;
            while (*vgen == gen) {
                if (*verr) break;
                if (((++it) & 1023u) == 0 && global_ns() - t0 > limit) {
                    atomicExch(bar + 2, 1u);
                    break;
                }
                __nanosleep(20);
            }
        }
        __threadfence();
        s_ok = (*verr == 0u);
    }
    __syncthreads();
    return s_ok != 0;
}

// ---- grid-wide sums that are the barrier as well
//
// A phase of the persistent kernels ends with every block publishing its partial sums and
// every block reading all of them: nobody can have them all before everybody has arrived,
// so reading the sums IS the barrier.  Against a counter and a second read of the partials
// this saves the serialised atomics of 148 blocks and one L2 round trip per phase (FP32
// sphere solve, 450k contacts: see k_apgd_sph for both sides measured).
//
// A slot holds 8 doubles per block; an unpublished value is all ones bits (a NaN that
// publish() never writes).  Phase m uses slot m & 3, and at phase m a block empties its own
// record of slot (m + 2) & 3: it was last read in phase m - 2, and this block has passed
// phase m - 1, which every block enters only after its phase m - 2 reads.  The emptied
// record is ordered before this block's next publication by the fence of publish().
// The host sets all slots to all ones before the launch.
constexpr int kSumSlots = 4;
constexpr int kSumRec = 8;
constexpr int kSumMaxBlocks = 160;  // five records per lane of the collecting warp

__device__ __forceinline__ double sum_empty() { return __longlong_as_double(-1ll); }
__device__ __forceinline__ bool sum_is_empty(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_relaxed_f64(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ double ld_relaxed_f64(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ld_relaxed_2f64(const double* p, double& a, double& b) {
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p) : "memory");
}

template <int NP>
struct SumShift {
    // lanes per value of multi_reduce<NP> (NP = 1, 2, 4 or 8), as a shift
    static constexpr int value = NP == 1 ? 5 : NP == 2 ? 4 : NP == 4 ? 3 : 2;
};
// Sums of NP values over the warp: lane l returns the sum of value l >> SumShift<NP>.  Each
// exchange halves the values a lane carries (9 shuffles for 8 values instead of 40); the
// additions are those of a shfl_down tree over lanes (+16, +8, +4, +2, +1), pair by pair.
template <int NP>
__device__ __forceinline__ double multi_reduce(double* v) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int h = NP / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = up ? v[i] : v[i + h];
            const double keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double x = v[0];
#pragma unroll
    for (; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Value k of this block's record for phase m (called by whole warp 0; `holds` marks the lanes
// with a value).  Everything the block wrote before the block barrier that precedes the call
// is visible to whoever collects the record (fence, then relaxed stores).
__device__ __forceinline__ void sum_publish(double* slots, unsigned int nb, unsigned int m, bool holds, int k, double v,
                                            bool withhold) {
    const size_t rec = (size_t)blockIdx.x * kSumRec + k;
    if (holds) st_relaxed_f64(slots + (size_t)((m + 2) & 3) * nb * kSumRec + rec, sum_empty());
    fence_gpu();
    if (holds && !withhold)
        st_relaxed_f64(slots + (size_t)(m & 3) * nb * kSumRec + rec, v == v ? v : __longlong_as_double(0x7ff8000000000000ll));
}

// The NP values of NW groups of 32 blocks from block b0 on (all of them: NW = 5, b0 = 0;
// nb <= kSumMaxBlocks): lane l gets blocks b0 + l, b0 + l + 32, ... in x (zeros past nb).  Called
// by one whole warp.  A wait longer than the limit (bar[3]) sets the error flag bar[2]; every
// waiter sees the flag and returns false.
template <int NP, int NW>
__device__ __forceinline__ bool sum_collect(const double* slots, unsigned int nb, unsigned int m, unsigned int* bar,
                                            double (&x)[NW][NP], unsigned int b0 = 0) {
    const unsigned int lane = b0 + (threadIdx.x & 31);
    const double* base = slots + (size_t)(m & 3) * nb * kSumRec;
    unsigned int pending = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
#pragma unroll
        for (int k = 0; k < NP; ++k) x[w][k] = 0.0;
        if (lane + 32u * w < nb) pending |= 1u << w;
    }
    const unsigned long long limit = barrier_limit_ns(bar);
    unsigned long long t0 = 0;
    bool ok = true;
    for (unsigned int it = 1;; ++it) {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if (!(pending & (1u << w))) continue;
            const double* r = base + (size_t)(lane + 32u * w) * kSumRec;
            if (NP == 1) {
                x[w][0] = ld_relaxed_f64(r);
            } else {
#pragma unroll
                for (int k = 0; k + 1 < NP; k += 2) ld_relaxed_2f64(r + k, x[w][k], x[w][k + 1]);
            }
        }
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if (!(pending & (1u << w))) continue;
            bool got = true;
#pragma unroll
            for (int k = 0; k < NP; ++k) got = got && !sum_is_empty(x[w][k]);
            if (got) pending &= ~(1u << w);
        }
        if (__all_sync(0xffffffffu, pending == 0)) break;
        if ((it & 63u) == 0) {
            const unsigned long long t = global_ns();
            bool late = *(volatile unsigned int*)(bar + 2) != 0u;
            if (t0 == 0) {
                t0 = t;
            } else if (t - t0 > limit) {
                atomicExch(bar + 2, 1u);
                late = true;
            }
            if (__any_sync(0xffffffffu, late)) {
                ok = false;
                break;
            }
        }
        if (it > 8) __nanosleep(32);
    }
    fence_gpu();
    return ok;
}
// Orders of the grid sum.  Lane order: lane l adds its blocks l, l + 32, ..., then the tree
// over lanes.  Group order: a tree per 32 consecutive blocks, then the groups in order.  Both
// give lane l the total of value l >> SumShift<NP>, the same bits in every block.
template <int NP>
__device__ __forceinline__ double sum_lane_order(const double (&x)[5][NP]) {
    double t[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        t[k] = 0.0;
#pragma unroll
        for (int w = 0; w < 5; ++w) t[k] += x[w][k];
    }
    return multi_reduce<NP>(t);
}
template <int NP>
__device__ __forceinline__ double sum_group_order(double (&x)[5][NP]) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 5; ++w) s += multi_reduce<NP>(x[w]);
    return s;
}

// (The kernels with one exchange per iteration reduce the contact sums over the warps while the
// barrier between the passes waits, and one more value after the particle pass.)
// Block partials of NP per-thread values, first half: per-warp sums into sh[k][warp].  After a
// block barrier, warp 0 finishes with block_sums_tree (tree over warps) or
// block_sums_in_order (warps one after the other); lane l gets value l >> SumShift<NP>.
template <int NP>
__device__ __forceinline__ void warp_sums(double* v, double (*sh)[32]) {
    const int lane = threadIdx.x & 31;
    const double x = multi_reduce<NP>(v);
    if ((lane & ((1 << SumShift<NP>::value) - 1)) == 0) sh[lane >> SumShift<NP>::value][threadIdx.x >> 5] = x;
}
__device__ __forceinline__ void warp_sum_to(double v, double* sh) {
    const double x = multi_reduce<1>(&v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
}
template <int NP>
__device__ __forceinline__ double block_sums_tree(const double (*sh)[32]) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double v[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) v[k] = lane < nw ? sh[k][lane] : 0.0;
    return multi_reduce<NP>(v);
}

// Fixed-order sum of NP doubles over the block (up to 1024 threads); the result is
// returned in every thread.
template <int NP>
__device__ __forceinline__ void block_sum(double* v) {
    __shared__ double sh[32][NP];
    __shared__ double tot[NP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < NP) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += sh[w][threadIdx.x];
        tot[threadIdx.x] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NP; ++k) v[k] = tot[k];
    __syncthreads();
}

// Block sum whose result only thread 0 needs (it is in thread 0's v[] on return): one
// block barrier.  The caller synchronises the block before the next call, which reuses
// the staging array.  Fixed summation order (deterministic).
template <int NP>
__device__ __forceinline__ void block_reduce_t0(double* v) {
    __shared__ double sh[NP][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[k][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            double x = lane < nw ? sh[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            v[k] = x;
        }
    }
}

// The sums of one phase after the other over the grid (every block of a cooperative launch).
// publish: all threads, their NP values; collect: warp 0, the totals in every lane; next: all
// threads, once per phase.  TREE: block sums as a tree over warps and lane order over blocks;
// else warps one after the other and group order over blocks (each solve keeps one order, so
// that its FP64 decisions do not depend on the launch).
template <bool TREE>
struct GridSums {
    double* slots;
    unsigned int nb;
    unsigned int* bar;
    unsigned int m;   // phase
    bool withhold;    // test of the wait limit: this block never publishes its first phase

    template <int NP>
    __device__ __forceinline__ void publish(double* v, double (*sh)[32]) {
        static_assert(TREE, "the streaming form's sums");
        warp_sums<NP>(v, sh);
        publish_warps<NP>(sh);
    }
    template <int NP>
    __device__ __forceinline__ void publish_warps(double (*sh)[32]) {
        __syncthreads();
        if (threadIdx.x < 32) {
            if (TREE) {
                constexpr int sf = SumShift<NP>::value;
                const double x = block_sums_tree<NP>(sh);
                sum_publish(slots, nb, m, (threadIdx.x & ((1 << sf) - 1)) == 0, threadIdx.x >> sf, x,
                            withhold && m == 0);
            } else {
                double x = 0.0;
                if (threadIdx.x < NP)
                    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += sh[threadIdx.x][w];
                sum_publish(slots, nb, m, threadIdx.x < NP, threadIdx.x, x, withhold && m == 0);
            }
        }
    }
    template <int NP>
    __device__ __forceinline__ bool collect(double* t) {
        static_assert(TREE, "the streaming form's sums");
        double x[5][NP];
        const bool ok = sum_collect<NP, 5>(slots, nb, m, bar, x);
        const double y = sum_lane_order<NP>(x);
#pragma unroll
        for (int k = 0; k < NP; ++k) t[k] = __shfl_sync(0xffffffffu, y, k << SumShift<NP>::value);
        return ok;
    }
    __device__ __forceinline__ void next() { ++m; }
    // a barrier without sums, split so that work can be done between the halves (all threads)
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        if (threadIdx.x < 32) sum_publish(slots, nb, m, threadIdx.x == 0, 0, 0.0, withhold && m == 0);
    }
    __device__ __forceinline__ bool wait() {
        __shared__ int s_ok;
        if (threadIdx.x < 32) {
            double x[5][1];
            const bool ok = sum_collect<1, 5>(slots, nb, m, bar, x);
            if (threadIdx.x == 0) s_ok = ok;
        }
        ++m;
        __syncthreads();
        return s_ok != 0;
    }
    // publish and collect in one, from the per-warp sums in sh (all threads, at least 160; the
    // totals and the status are warp 0's).  Five warps collect a group of blocks each, so that no thread holds more than NP of
    // the values.
    template <int NP>
    __device__ __forceinline__ bool sums(double (*sh)[32], double* t) {
        __shared__ double raw[5][NP][32];
        __shared__ int bad;
        if (threadIdx.x == 0) bad = 0;
        publish_warps<NP>(sh);
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (w < 5) {
            double x[1][NP];
            const bool ok = sum_collect<NP, 1>(slots, nb, m, bar, x, 32u * w);
            if (TREE) {
#pragma unroll
                for (int k = 0; k < NP; ++k) raw[w][k][lane] = x[0][k];
            } else {
                const double z = multi_reduce<NP>(x[0]);
                if ((lane & ((1 << SumShift<NP>::value) - 1)) == 0) raw[w][lane >> SumShift<NP>::value][0] = z;
            }
            if (!ok && lane == 0) bad = 1;
        }
        ++m;
        __syncthreads();
        if (w == 0 && !TREE) {
            double z = 0.0;
            if (lane < NP)
#pragma unroll
                for (int g = 0; g < 5; ++g) z += raw[g][lane][0];
#pragma unroll
            for (int k = 0; k < NP; ++k) t[k] = __shfl_sync(0xffffffffu, z, k);
        } else if (w == 0) {
            double y[NP];
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                y[k] = 0.0;
#pragma unroll
                for (int g = 0; g < 5; ++g) y[k] += raw[g][k][lane];
            }
            const double z = multi_reduce<NP>(y);
#pragma unroll
            for (int k = 0; k < NP; ++k) t[k] = __shfl_sync(0xffffffffu, z, k << SumShift<NP>::value);
        }
        return bad == 0;
    }
    __device__ __forceinline__ void finish() {}
    // one value per block (the same in all its threads), summed in group order; a full barrier
    __device__ __forceinline__ bool exchange(double v, double& total) {
        __shared__ double s_t;
        __shared__ int s_ok;
        __syncthreads();
        if (threadIdx.x < 32) {
            sum_publish(slots, nb, m, threadIdx.x == 0, 0, v, withhold && m == 0);
            double x[5][1];
            const bool ok = sum_collect<1, 5>(slots, nb, m, bar, x);
            const double y = sum_group_order<1>(x);
            if (threadIdx.x == 0) {
                s_t = y;
                s_ok = ok;
            }
        }
        ++m;
        __syncthreads();
        total = s_t;
        return s_ok != 0;
    }
};

// roundings written out where the compiler could contract in more than one way: a solve's
// bits are then the same whatever kernel it runs in
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// LagrangeMultiplier<Friction>::projection, include/scopi/solvers/lagrange_multiplier.hpp:243-268
template <int DIM>
__device__ __forceinline__ void cone_project(double* l, const double* n, double mu) {
    double ln = 0.0;
    for (int d = 0; d < DIM; ++d) ln += l[d] * n[d];
    double lt[3] = {0, 0, 0};
    for (int d = 0; d < DIM; ++d) lt[d] = l[d] - ln * n[d];
    double nrm = 0.0;
    for (int d = 0; d < DIM; ++d) nrm += lt[d] * lt[d];
    nrm = sqrt(nrm);
    if (nrm > mu * ln) {
        if (ln <= -mu * nrm) {
            for (int d = 0; d < DIM; ++d) l[d] = 0.0;
        } else {
            const double nn = (mu * mu) * (nrm + ln / mu) / (mu * mu + 1);
            const double nln = nn / mu;
            for (int d = 0; d < DIM; ++d) l[d] = nn * (lt[d] / nrm) + nln * n[d];
        }
    }
}

// Backtracking test of apgd.hpp:172-182, F(l+) >= F(y) + g(y).d + L/2 |d|^2 with d = l+ - y.
// FP64 evaluates it as the reference does.  For a quadratic F the test is exactly
// d^T Q d >= L |d|^2; FP32 iterations use that form (dQd = dt^2 sum_p m |u(l+) - u(y)|^2),
// since F(l+) - F(y) in FP32 carries round-off of the size of F itself and fails the
// test spuriously once the steps are small, which collapses alpha and stalls the solve.
template <typename T>
__device__ __forceinline__ bool sufficient_decrease_fails(double F_lp, double Fy, double gd, double dd, double dQd,
                                                          double lipsch) {
    if (sizeof(T) == 4) return dQd >= lipsch * dd;
    return F_lp >= Fy + gd + 0.5 * lipsch * dd;
}

// First projected-gradient direction of a solve at its cold start (lambda = 0, or delta = 0
// for a correction with offset `shift`): d = -g where the bound lets it move.  The
// Rayleigh quotient d^T Q d / |d|^2 then sets the initial step (see the kernels).
template <typename T>
__device__ __forceinline__ T first_descent(T g, const double* shift, long long m) {
    if (shift) return (shift[m] > 0.0 || g < (T)0) ? -g : (T)0;
    return g < (T)0 ? -g : (T)0;
}
// Initial Lipschitz estimate: 1.5 x the curvature along d (d^T Q d = dt^2 sum_p
// w_p . M^-1 w_p with w = B^T d).  The reference starts every solve from the fixed
// alpha = 0.05 (apgd.hpp:120) and grows it by 1/0.97 per accepted iteration; for the
// problems here 1/L is many orders of magnitude larger, so most of its iterations are
// that ramp, and its first step alpha*|g| can fall below the tolerance so that the solve
// stops at once with a resting contact still open by ~ g dt^2.
__device__ __forceinline__ bool initial_lipschitz(double dd, double wmw, double dt2, double& lipsch) {
    if (!(dd > 0.0) || !(wmw > 0.0)) return false;
    const double l = 1.5 * dt2 * wmw / dd;
    if (!isfinite(l) || !(l > 0.0)) return false;
    lipsch = l;
    return true;
}

// l+ == y bit for bit: the reference compares F(l+) >= F(y) on identical vectors, doubles
// L (l+ cannot move: -g lies in the normal cone at y) until 0.5*L*0 turns NaN at L = inf,
// then accepts with alpha = 0 (apgd.hpp:172-182).
__device__ __forceinline__ void overflow_cascade(double& lipsch, double& alpha, long long& nbt) {
    while (isfinite(lipsch)) {
        lipsch *= 2;
        ++nbt;
    }
    alpha = 1. / lipsch;
}

// The same for a launch of one cluster (up to 16 CTAs): hardware cluster barriers, block sums
// read through distributed shared memory, in the orders of GridSums<TREE>.  Nothing can be
// missing from such a barrier (the CTAs of a cluster run together), so there is no limit.
template <bool TREE>
struct ClusterSums {
    int par;

    // an aligned barrier wants whole warps: lanes that took different branches meet first
    __device__ __forceinline__ void arrive() {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    __device__ __forceinline__ bool wait() {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    __device__ __forceinline__ static double remote(const double* own, unsigned int rank) {
        const unsigned int a = (unsigned int)__cvta_generic_to_shared(own);
        unsigned int r;
        double v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(r) : "memory");
        return v;
    }
    // a slot is written again two exchanges later, when every CTA has passed the barrier of the
    // exchange between, which it enters after its reads
    template <int NP>
    __device__ __forceinline__ void read(const double* own, double (&x)[1][NP]) {
        const unsigned int lane = threadIdx.x & 31;
#pragma unroll
        for (int k = 0; k < NP; ++k) x[0][k] = lane < gridDim.x ? remote(own + k, lane) : 0.0;
    }
    template <int NP>
    __device__ __forceinline__ bool sums(double (*sh)[32], double* t) {
        __shared__ double part[2][8];
        __syncthreads();
        constexpr int sf = SumShift<NP>::value;
        if (threadIdx.x < 32) {
            if (TREE) {
                const double x = block_sums_tree<NP>(sh);
                if ((threadIdx.x & ((1 << sf) - 1)) == 0) part[par][threadIdx.x >> sf] = x;
            } else if (threadIdx.x < NP) {
                double x = 0.0;
                for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += sh[threadIdx.x][w];
                part[par][threadIdx.x] = x;
            }
        }
        arrive();
        wait();
        if (threadIdx.x < 32) {
            double x[1][NP];
            read<NP>(part[par], x);
            // one group of at most 16 blocks: both orders are its tree
            const double y = multi_reduce<NP>(x[0]);
#pragma unroll
            for (int k = 0; k < NP; ++k) t[k] = __shfl_sync(0xffffffffu, y, k << sf);
        }
        par ^= 1;
        return true;
    }
    __device__ __forceinline__ bool exchange(double v, double& total) {
        __shared__ double one[2];
        __shared__ double s_t;
        if (threadIdx.x == 0) one[par] = v;
        arrive();
        wait();
        if (threadIdx.x < 32) {
            double x[1][1];
            read<1>(&one[par], x);
            const double y = multi_reduce<1>(x[0]);
            if (threadIdx.x == 0) s_t = y;
        }
        par ^= 1;
        __syncthreads();
        total = s_t;
        return true;
    }
    // before a CTA leaves: nobody reads its shared memory any more
    __device__ __forceinline__ void finish() {
        arrive();
        wait();
    }
};

template <bool CL, bool TREE>
struct SyncOf;
template <bool TREE>
struct SyncOf<false, TREE> {
    using type = GridSums<TREE>;
};
template <bool TREE>
struct SyncOf<true, TREE> {
    using type = ClusterSums<TREE>;
};
template <bool TREE>
__device__ __forceinline__ void sync_init(GridSums<TREE>& G, double* slots, unsigned int* bar, bool stall) {
    G = GridSums<TREE>{slots, gridDim.x, bar, 0u, stall};
}
template <bool TREE>
__device__ __forceinline__ void sync_init(ClusterSums<TREE>& G, double*, unsigned int*, bool) {
    G.par = 0;
}

// Host: whether the current device can run `kernel` as one cluster of 2^lg CTAs (0 not asked, 1 yes,
// 2 no).  The permission for clusters of more than 8 belongs to the kernel on one device, so each
// device of the process is asked for itself; devices past kMaxDevices take the cooperative launch.
constexpr int kMaxCluster = 16;
struct ClusterAble {
    std::atomic<int> at[kMaxDevices][5];  // [device][lg], lg <= 4
};
inline cudaLaunchConfig_t cluster_config(int n, int threads, cudaStream_t s, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = n;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}
template <typename K>
bool cluster_fits(K kernel, const cudaLaunchConfig_t& cfg, ClusterAble& known, int lg) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
    std::atomic<int>& able = known.at[dev][lg];
    int a = able.load(std::memory_order_relaxed);
    if (a == 0) {
        int fit = 0;
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0;
        if (!ok) cudaGetLastError();
        a = ok ? 1 : 2;
        able.store(a, std::memory_order_relaxed);
    }
    return a == 1;
}
inline int log2_up(int n) {
    int lg = 0;
    while ((1 << lg) < n) ++lg;
    return lg;
}

// Loop-carried scalars of the iteration (block-uniform) live in shared memory and are
// updated by thread 0, so the registers go to the two passes.
struct ApgdState {
    double alpha, lipsch, theta, beta, beta_n, theta1, Fy, last_step, lgood;
    double tk[4];  // g.d, |d|^2, c.l+ and |l+|^2 of the candidate (contact pass sums)
    long long ite, nbt, nrs;
    int il, ip, in_, jL, jN, jY, jYN, bt, use_prev, restart, done, conv, err;
};
__device__ __forceinline__ void state_init(ApgdState& S, double alpha) {
    S.alpha = alpha;
    S.lipsch = 1.0 / alpha;
    S.lgood = S.lipsch;
    S.theta = 1.0;
    S.beta = 0.0;
    S.beta_n = 0.0;
    S.theta1 = 1.0;
    S.Fy = 0.0;
    S.last_step = 0.0;
    S.ite = S.nbt = S.nrs = 0;
    S.il = 0; S.ip = 1; S.in_ = 2;           // lambda buffers: current, previous, candidate
    S.jL = 0; S.jN = 1; S.jY = 2; S.jYN = 3;  // u buffers: u(l), u(candidate), u(y), u(next y)
    S.bt = 0;
    S.use_prev = 0;
    S.restart = 0;
    S.done = 0;
    S.conv = 0;
    S.err = 0;
}

// The two decisions of an iteration, taken by thread 0 of every block from the same sums.
// What does not depend on the sums (momentum, both candidate steps, square roots) is computed
// by prepare_* while the sums are still on their way.
struct Momentum {
    double theta1, beta;
};
__device__ __forceinline__ Momentum prepare_momentum(const ApgdState& S) {
    const double th = S.theta, t2 = mul_rn(th, th);
    Momentum m;
    m.theta1 = 0.5 * fma_rn(th, sqrt(add_rn(4.0, t2)), -t2);
    m.beta = mul_rn(th, add_rn(1.0, -th)) / add_rn(t2, m.theta1);
    return m;
}
// after the contact pass: momentum for the next y if this candidate is accepted
// (apgd.hpp:196-206); t: FP64 g.d, |d|^2, c.l+, F(y), |l+ - l|^2, g.(l+ - l), |l+|^2;
// FP32 |d|^2, |l+ - l|^2, g.(l+ - l), |l+|^2
template <typename T>
__device__ __forceinline__ void decide_momentum(ApgdState& S, const double* t, bool bt, int dynamic, Momentum m) {
    constexpr bool f32 = sizeof(T) == 4;
    S.theta1 = m.theta1;
    S.restart = (dynamic && t[f32 ? 2 : 5] > 0) ? 1 : 0;
    S.beta_n = S.restart ? 0.0 : m.beta;
    if (!f32 && !bt) S.Fy = t[f32 ? 0 : 3];
    // the scalars the decision needs after the second pass
    S.last_step = t[f32 ? 1 : 4];
    S.tk[0] = f32 ? 0.0 : t[0];
    S.tk[1] = t[f32 ? 0 : 1];
    S.tk[2] = f32 ? 0.0 : t[f32 ? 0 : 2];
    S.tk[3] = t[f32 ? 3 : 6];
}
struct NextStep {
    double tol, step, alpha_bt, lip_ok, alpha_ok;
};
template <typename T>
__device__ __forceinline__ NextStep prepare_step(const ApgdState& S, double tol) {
    NextStep n;
    n.tol = tol;
    if (sizeof(T) == 4) {
        // FP32 iterations stall at their rounding floor; the FP64 correction recovers the rest
        const double floor32 = 4.0 * 1.1920929e-7 * sqrt(S.tk[3]);
        if (floor32 > n.tol) n.tol = floor32;
    }
    n.step = sqrt(S.last_step);
    n.alpha_bt = 1. / (S.lipsch * 2);
    n.lip_ok = S.lipsch * 0.97;
    n.alpha_ok = 1. / n.lip_ok;
    return n;
}
// the same once the sums are known: sq = sqrt(|l+ - l|^2), sq1 = sqrt(|l+|^2)
template <typename T>
__device__ __forceinline__ NextStep step_of(NextStep n, double tol, double sq, double sq1) {
    n.step = sq;
    n.tol = tol;
    if (sizeof(T) == 4) {
        const double floor32 = 4.0 * 1.1920929e-7 * sq1;
        if (floor32 > n.tol) n.tol = floor32;
    }
    return n;
}
// after the particle pass: backtrack or accept (apgd.hpp:172-221); wu = w.u (FP64), curv =
// |u(l+) - u(y)|^2_M (FP32); more than max_bt backtracks (0: no limit) end the solve with error 2
template <typename T>
__device__ __forceinline__ void decide_step(ApgdState& S, double wu, double curv, double dt2, int dynamic,
                                            long long max_ite, NextStep n, long long max_bt = 0) {
    const double* tk = S.tk;
    const double F_lp = 0.5 * dt2 * wu + tk[2];
    if (dynamic && tk[1] == 0.0) {
        double lip = S.lipsch, al = S.alpha;
        long long nbt = S.nbt;
        overflow_cascade(lip, al, nbt);
        S.lipsch = lip;
        S.alpha = al;
        S.nbt = nbt;
        n.lip_ok = lip * 0.97;
        n.alpha_ok = 1. / n.lip_ok;
    } else if (dynamic && sufficient_decrease_fails<T>(F_lp, S.Fy, tk[0], tk[1], dt2 * curv, S.lipsch)) {
        S.lipsch *= 2;  // backtracking, apgd.hpp:172-182
        S.alpha = n.alpha_bt;
        S.bt = 1;
        ++S.nbt;
        if (max_bt > 0 && S.nbt > max_bt) {  // alpha underflow guard
            S.err = 2;
            S.done = 1;
        }
        return;
    }
    ++S.ite;
    S.bt = 0;
    if (isfinite(S.lipsch)) S.lgood = S.lipsch;
    S.last_step = n.step;
    int tmp = S.ip; S.ip = S.il; S.il = S.in_; S.in_ = tmp;
    tmp = S.jL; S.jL = S.jN; S.jN = tmp;
    tmp = S.jY; S.jY = S.jYN; S.jYN = tmp;
    if (n.step < n.tol) {
        S.conv = 1;
        S.done = 1;
        return;
    }
    S.beta = S.beta_n;
    S.theta = S.restart ? 1.0 : S.theta1;
    if (S.restart) ++S.nrs;
    if (dynamic) {
        S.lipsch = n.lip_ok;
        S.alpha = n.alpha_ok;
    }
    S.use_prev = (S.beta != 0.0) ? 1 : 0;
    if (S.ite >= max_ite) S.done = 1;
}
// After an accepted step of the kernels whose particle pass does not wait for the sums: a
// restart makes u(l+) the next u(y); the candidates take the two free buffers.
__device__ __forceinline__ void reuse_buffers(ApgdState& S) {
    if (S.restart) S.jY = S.jL;
    int free[2] = {0, 0}, n = 0;
    for (int j = 0; j < 4 && n < 2; ++j)
        if (j != S.jL && j != S.jY) free[n++] = j;
    S.jN = free[0];
    S.jYN = free[1];
}
__device__ __forceinline__ void write_result(ApgdResult* r, const ApgdState& S) {
    r->iterations = S.ite;
    r->backtracks = S.nbt;
    r->restarts = S.nrs;
    r->converged = S.conv;
    r->lam_buf = S.il;
    r->u_buf = S.jL;
    r->error = S.err;
    r->last_step = S.last_step;
    r->lipsch = S.lgood;
}

}  // namespace apgdc
}  // namespace scopi_gpu
