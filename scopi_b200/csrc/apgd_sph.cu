// apgd_sph.cu -- persistent APGD for the normal-only problems (NoFriction, Viscous) on
// contacts whose lever arms are parallel to the normal (sphere-sphere, sphere-plane,
// sphere-segment: p_i - x_i = -/+ r_i n), where the rotational terms of the contact
// Jacobian, R^T (r x n), vanish identically.  A contact's row of B is then n^T on the
// two bodies' translational velocities:
//     (B u)_c = n_c . (u_i - u_j),     (B^T l)_p = sum_{c ~ p} +-l_c n_c.
// Same iteration, branch logic and stopping rule as the generic kernel (apgd.cu), i.e.
// apgd::operator() of include/scopi/solvers/apgd.hpp:148-221, with the data cut to
// what this row shape needs:
//   per contact : (ci, cj) int2 + (n, c) packed in one 16/32-byte record, l, l_prev;
//   per incidence of a body: (+-n, contact index) in one record;
//   per body    : u(y) gathered once (u(y_next) = u(l+) + beta (u(l+) - u(l)) is formed in
//                 the particle pass, the restart test being reduced after the first barrier).
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "../../include/scopi_gpu.h"
#include "apgd_common.cuh"

namespace scopi_gpu {

static long long g_sph_launches = 0;
long long apgd_sph_launches() { return g_sph_launches; }

namespace {
using namespace apgdc;

__device__ __forceinline__ float4 ld4(const float4* p) { return *p; }
__device__ __forceinline__ dvec4 ld4(const dvec4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = q[0], b = q[1];
    return dvec4{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void st4(float4* p, float x, float y, float z) { *p = make_float4(x, y, z, 0.f); }
__device__ __forceinline__ void st4(dvec4* p, double x, double y, double z) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0] = make_double2(x, y);
    q[1] = make_double2(z, 0.0);
}
// incidence record r of a body: (+-n, contact index)
__device__ __forceinline__ float4 ld_inc(const float4* inc, const IncWalk& w, int r) { return inc[w.first + (long long)r * w.rs]; }
__device__ __forceinline__ dvec4 ld_inc(const double2* inc, const IncWalk& w, int r) {
    const double2* q = inc + w.first + (long long)r * w.rs;
    const double2 a = q[0], b = q[w.vs];
    return dvec4{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ int idx_of(float w) { return __float_as_int(w); }
__device__ __forceinline__ int idx_of(double w) { return (int)__double_as_longlong(w); }

// ---- asynchronous global -> shared copies (cp.async).  Each thread stages only the
// records it consumes itself, so a stage needs no block barrier: cp.async.wait_group
// makes the thread's own copies visible to it.  src-size 0 zero-fills the slot without
// reading (tails past the end; the source pointer is then the array base).
__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void* dst, const void* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sm_addr(dst)), "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}
// the same with an L2 eviction policy
__device__ __forceinline__ void cp16h(void* dst, const void* src, bool on, unsigned long long pol) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(sm_addr(dst)), "l"(src),
                 "r"(on ? 16 : 0), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void cp8h(void* dst, const void* src, bool on, unsigned long long pol) {
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 8, %2, %3;\n" ::"r"(sm_addr(dst)), "l"(src),
                 "r"(on ? 8 : 0), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void cp_vech(float4* d, const float4* s, bool on, unsigned long long pol) { cp16h(d, s, on, pol); }
__device__ __forceinline__ void cp_vech(dvec4* d, const dvec4* s, bool on, unsigned long long pol) {
    cp16h(d, s, on, pol);
    cp16h(reinterpret_cast<double2*>(d) + 1, reinterpret_cast<const double2*>(s) + 1, on, pol);
}
__device__ __forceinline__ unsigned long long evict_first_policy() {
    unsigned long long p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// incidence record r of a body with that policy (the records do not change during the solve)
__device__ __forceinline__ float4 ld_inch(const float4* inc, const IncWalk& w, int r, unsigned long long pol) {
    float4 v;
    asm("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(inc + w.first + (long long)r * w.rs), "l"(pol));
    return v;
}
__device__ __forceinline__ dvec4 ld_inch(const double2* inc, const IncWalk& w, int r, unsigned long long pol) {
    const double2* q = inc + w.first + (long long)r * w.rs;
    dvec4 v;
    asm("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(q), "l"(pol));
    asm("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.z), "=d"(v.w) : "l"(q + w.vs), "l"(pol));
    return v;
}
__device__ __forceinline__ void cp8(void* dst, const void* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sm_addr(dst)), "l"(src), "r"(on ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sm_addr(dst)), "l"(src), "r"(on ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_val(float* d, const float* s, bool on) { cp4(d, s, on); }
__device__ __forceinline__ void cp_val(double* d, const double* s, bool on) { cp8(d, s, on); }
__device__ __forceinline__ void cp_vec(float4* d, const float4* s, bool on) { cp16(d, s, on); }
__device__ __forceinline__ void cp_vec(dvec4* d, const dvec4* s, bool on) {
    cp16(d, s, on);
    cp16(reinterpret_cast<double2*>(d) + 1, reinterpret_cast<const double2*>(s) + 1, on);
}

template <typename T>
struct SphArgs {
    int nin, na;
    const int2* cij;
    const V4<T>* nc;
    const int* slot;
    const double* shift;
    const int* inc_ptr;
    const Q16<T>* inc;
    long long inc_slots;
    const T* invm;  // 1/m per active body, contiguous
    T* lam0;
    T* lam1;
    T* lam2;
    V4<T>* u0;
    V4<T>* u1;
    V4<T>* u2;
    V4<T>* u3;
    double* sums;  // kSumSlots x blocks x kSumRec, all ones at launch
    unsigned int* bar;
    ApgdResult* result;
    const Sizes* sizes;
    double alpha, tol, dt2;
    long long max_ite;
    int dynamic;
    int curvature_start;
    int stall;  // block 0 skips its first barrier arrival (test of the barrier limit)
};

template <typename T>
__device__ __forceinline__ T pick(int k, T a, T b, T c) {
    return k == 0 ? a : (k == 1 ? b : c);
}
template <typename T>
__device__ __forceinline__ T pick4(int k, T a, T b, T c, T d) {
    return k == 0 ? a : (k == 1 ? b : (k == 2 ? c : d));
}

// n.u, rounded as the streaming pass rounds it
template <typename T, int DIM>
__device__ __forceinline__ T normal_dot(const V4<T>& n, const V4<T>& u) {
    const T xy = fma_rn(n.x, u.x, mul_rn(n.y, u.y));
    return DIM == 3 ? fma_rn(n.z, u.z, xy) : xy;
}
// one multiplier of the contact pass (lm, lpm: its current and previous values); returns l+
template <typename T>
__device__ __forceinline__ T mult_update_v(const SphArgs<T>& A, long long m, T qy, T gm, T cc, T lm, T lpm, T* lnew,
                                              T beta, bool use_prev, bool bt, double alpha, double* s) {
    const T y = use_prev ? fma_rn(beta, add_rn(lm, -lpm), lm) : lm;
    T lp;
    if (A.shift) {
        const double sh = A.shift[m];
        double z = sh + ((double)y - alpha * (double)gm);
        z = z > 0.0 ? z : 0.0;
        lp = (T)(z - sh);
    } else {
        const T z = fma_rn(-(T)alpha, gm, y);
        lp = z > (T)0 ? z : (T)0;
    }
    lnew[m] = lp;
    const double dly = (double)lp - (double)y, dll = (double)lp - (double)lm;
    // g.d, c.l+ and F(y) serve the reference's backtracking test (FP64 only; the FP32 test
    // is the curvature form, which reads |d|^2 and the particle pass's d^T Q d)
    if (sizeof(T) == 8) {
        s[0] += (double)gm * dly;
        s[2] += (double)cc * (double)lp;
        if (!bt) s[3] += (double)y * (0.5 * (double)qy + (double)cc);
    }
    s[1] += dly * dly;
    s[4] += dll * dll;
    s[5] += (double)gm * dll;
    s[6] += (double)lp * (double)lp;
    return lp;
}
// A contact: its row, u(y) of its bodies, the current and previous multipliers (lm2, lpm2: of the
// viscous second multiplier at slot sv, if any); returns the candidate(s).
template <typename T, int DIM, int PROB>
__device__ __forceinline__ T contact_update(const SphArgs<T>& A, long long c, const V4<T>& nc, const V4<T>& ui,
                                            const V4<T>& uj, T lm, T lpm, int sv, T lm2, T lpm2, T* lp2, T* lnew,
                                            T beta, bool use_prev, bool bt, double alpha, double* s) {
    // obstacles have u = 0
    const T q0 = add_rn(normal_dot<T, DIM>(nc, ui), -normal_dot<T, DIM>(nc, uj));
    const T qy = mul_rn(q0, (T)A.dt2);
    // one rounding where the product is wanted for nothing else
    const T gm = sizeof(T) == 4 && PROB == kNoFriction ? fma_rn(q0, (T)A.dt2, nc.w) : add_rn(qy, nc.w);
    const T lp = mult_update_v<T>(A, c, qy, gm, nc.w, lm, lpm, lnew, beta, use_prev, bt, alpha, s);
    if (PROB == kViscous && sv >= 0)
        *lp2 = mult_update_v<T>(A, sv, -qy, -gm, -nc.w, lm2, lpm2, lnew, beta, use_prev, bt, alpha, s);
    return lp;
}

// One block per SM (SphShape): FP32 768 threads (80 registers, no spills), FP64 512 (128).
// Chosen on the form with rows of incidence records, L2-only gathers and counter barriers, 1M
// spheres, 3.0M contacts, microseconds per iteration: FP32 70.6 against 77.1 with 1024 threads and
// the gathers one trip ahead; FP64 110.9 against 117.1, and 115.1 with 5 contact stages (shared
// memory and L1 share the SM, and the gathers live in L1).
//
// Each pass ends in grid sums that serve as the barrier (GridSums).  Against a barrier counter,
// a second read of the partials and 40 shuffles per warp for eight sums, microseconds per
// iteration: FP32 450k contacts 18.4 -> 16.8, 4.6M 112.0 -> 108.4; FP64 2k contacts 12.5 -> 10.8,
// 133k 18.0 -> 16.0, 4.6M 197.5 -> 188.6 (same bits: the order of every sum is unchanged).
//
// Both passes stream their per-item records through a cp.async pipeline in dynamic shared
// memory (the passes are separated by grid barriers, so they share it):
//   contact pass, GC stages, per contact : (ci, cj), (n, c), l, l_prev  -- 32 B (FP32), 56 B (FP64)
//   particle pass, GP stages, per body   : inc_ptr[p], inc_ptr[p+1], 1/m, u(l) and (FP32) u(y)
// and the gathers that depend on a staged record (u(y) of the contact's bodies) are issued
// GD trips ahead.  The incidence records stay on plain loads.
// Gathers (u(y), l+) are plain loads: the acquire of the barrier before the pass empties the L1, so
// they are fresh, and bodies shared by neighbouring contacts and multipliers that share a sector
// then come from L1 (against L2-only loads, microseconds per iteration: FP64 4.6M contacts
// 172.3 -> 154.3, 133k 11.4 -> 10.5; FP32 451k 15.7 -> 14.7, 4.6M 99.1 -> 97.2).
// Launch shape per precision: threads per block, contact-pass stages GC (the u(y) gathers
// of trip k + GD are issued during trip k: an L2 round trip is about one trip long),
// particle-pass stages GP.
template <typename T>
struct SphShape;
template <>
struct SphShape<float> {
    static constexpr int threads = 768, GC = 5, GD = 2, GP = 4;
};
template <>
struct SphShape<double> {
    static constexpr int threads = 512, GC = 4, GD = 2, GP = 4;
};
template <typename T>
struct SphOcc {
    static constexpr int threads = SphShape<T>::threads;
    static constexpr int GC = SphShape<T>::GC, GD = SphShape<T>::GD, GP = SphShape<T>::GP;
    static constexpr size_t contact_bytes = (size_t)GC * threads * (sizeof(int2) + sizeof(V4<T>) + 2 * sizeof(T));
    static constexpr size_t particle_bytes =
        (size_t)GP * threads * ((sizeof(T) == 4 ? 2 : 1) * sizeof(V4<T>) + sizeof(T) + 2 * sizeof(int));
    static constexpr size_t smem = contact_bytes > particle_bytes ? contact_bytes : particle_bytes;
};

// Initial step from the curvature along the first descent direction d (stored in the candidate
// buffer, which the first contact pass overwrites).
template <typename T, int DIM, int PROB, typename SY>
__device__ __forceinline__ void curvature_step(const SphArgs<T>& A, int C, IncLayout lay, ApgdState& S, SY& G) {
    T* dbuf = A.lam2;
    double t1 = 0.0, t3 = 0.0;
    double a2[2] = {0.0, 0.0};
    GRID_STRIDE(c, C) {
        const T cc = ld4(A.nc + c).w;
        const T d = first_descent<T>(cc, A.shift, c);
        dbuf[c] = d;
        a2[0] += (double)d * (double)d;
        if (PROB == kViscous) {
            const int sl = A.slot[c];
            if (sl >= 0) {
                const T d2 = first_descent<T>(-cc, A.shift, sl);
                dbuf[sl] = d2;
                a2[0] += (double)d2 * (double)d2;
            }
        }
    }
    block_sum<2>(a2);
    bool ok = G.exchange(a2[0], t1);
    double wm[2] = {0.0, 0.0};
    if (ok) GRID_STRIDE(p, A.na) {
        T w0 = 0, w1 = 0, w2 = 0;
        const int k0 = A.inc_ptr[p], n = A.inc_ptr[p + 1] - k0;
        const IncWalk wk = inc_walk(lay, sizeof(T) / 4, p, k0);
        for (int k = 0; k < n; ++k) {
            const V4<T> e = ld_inc(A.inc, wk, k);
            const int ci = idx_of(e.w);
            T mu = __ldcg(dbuf + ci);
            if (PROB == kViscous) {
                const int sl = A.slot[ci];
                if (sl >= 0) mu -= __ldcg(dbuf + sl);
            }
            w0 += mu * e.x;
            w1 += mu * e.y;
            if (DIM == 3) w2 += mu * e.z;
        }
        const double im = (double)A.invm[p];
        wm[0] += im * ((double)w0 * w0 + (double)w1 * w1 + (double)w2 * w2);
    }
    block_sum<2>(wm);
    if (ok) ok = G.exchange(wm[0], t3);
    if (threadIdx.x == 0) {
        double l;
        if (ok && initial_lipschitz(t1, t3, A.dt2, l)) {
            S.lipsch = l;
            S.alpha = 1.0 / l;
            S.lgood = l;
        }
        if (!ok) {
            S.err = 1;
            S.done = 1;
        }
    }
    __syncthreads();
}

template <typename T, int DIM, int PROB, bool PAST_L2>
__global__ void __launch_bounds__(SphOcc<T>::threads, 1) k_apgd_sph(SphArgs<T> A) {
    __shared__ ApgdState S;
    extern __shared__ __align__(32) unsigned char sph_dyn[];
    constexpr int GC = SphOcc<T>::GC, GD = SphOcc<T>::GD, GP = SphOcc<T>::GP;
    static_assert(GD >= 1 && GD <= GC - 2, "the gathered records must be in the prologue's stages");
    const int NT = blockDim.x, tid = threadIdx.x;
    // contact-pass stages [GC][NT] of each field
    V4<T>* s_nc = reinterpret_cast<V4<T>*>(sph_dyn);
    int2* s_ij = reinterpret_cast<int2*>(s_nc + GC * NT);
    T* s_l = reinterpret_cast<T*>(s_ij + GC * NT);
    T* s_lp = s_l + GC * NT;
    // particle-pass stages [GP][NT] (same memory)
    V4<T>* s_ul = reinterpret_cast<V4<T>*>(sph_dyn);
    V4<T>* s_uy = s_ul + GP * NT;  // FP32 only
    T* s_im = reinterpret_cast<T*>(s_ul + (sizeof(T) == 4 ? 2 : 1) * GP * NT);
    int* s_p0 = reinterpret_cast<int*>(s_im + GP * NT);
    int* s_p1 = s_p0 + GP * NT;
    __shared__ double red[8][32];
    if (threadIdx.x == 0) state_init(S, A.alpha);
    __syncthreads();
    const int C = A.sizes->C;
    const IncLayout lay = inc_layout(A.sizes, A.na, A.inc_slots);
    // PAST_L2 (the solve does not fit the L2): what an iteration only streams, the rows and the
    // incidence records, leaves the L2 first, so that the multipliers and velocities that the
    // passes gather stay
    const unsigned long long pol = PAST_L2 ? evict_first_policy() : 0;
    GridSums<true> G{A.sums, gridDim.x, A.bar, 0u, A.stall != 0 && blockIdx.x == 0};
    // Trip k of a thread handles item base + k*S (the grid-stride order) in both passes.
    const long long S_ = (long long)gridDim.x * NT, base = (long long)blockIdx.x * NT + tid;
    const long long ntrip_c = ((long long)C - (long long)blockIdx.x * NT + S_ - 1) / S_;
    const long long ntrip_p = ((long long)A.na - (long long)blockIdx.x * NT + S_ - 1) / S_;
    // First stages of each pass are issued before the grid barrier that precedes the pass
    // when they do not depend on it: a contact's geometry (n, c), (ci, cj), and a body's
    // inc_ptr, 1/m, u(l), u(y).  Uncommitted copies join the next commit group.
    auto issue_geom = [&](int k) {
        const int sl = (k % GC) * NT + tid;
        const long long c = base + k * S_;
        const bool on = k < ntrip_c && c < C;
        const long long cc = on ? c : 0;
        if (PAST_L2) {
            cp_vech(s_nc + sl, A.nc + cc, on, pol);
            cp8h(s_ij + sl, A.cij + cc, on, pol);
        } else {
            cp_vec(s_nc + sl, A.nc + cc, on);
            cp8(s_ij + sl, A.cij + cc, on);
        }
    };
    auto issue_body = [&](long long k, const V4<T>* uL, const V4<T>* uY, bool with_ul) {
        const int sl = (int)(k % GP) * NT + tid;
        const long long p = base + k * S_;
        const bool on = k < ntrip_p && p < A.na;
        const long long pp = on ? p : 0;
        cp4(s_p0 + sl, A.inc_ptr + pp, on);
        cp4(s_p1 + sl, A.inc_ptr + pp + 1, on);
        cp_val(s_im + sl, A.invm + pp, on);
        cp_vec(s_ul + sl, uL + pp, on && with_ul);
        if (sizeof(T) == 4) cp_vec(s_uy + sl, uY + pp, on);
        cp_commit();
    };
    bool geom_issued = false;
    if (A.curvature_start) curvature_step<T, DIM, PROB>(A, C, lay, S, G);
    for (;;) {
        if (S.done) break;
        const double alpha = S.alpha;
        const bool bt = S.bt != 0, use_prev = S.use_prev != 0;
        const T beta = (T)S.beta;
        const T* lam = pick(S.il, A.lam0, A.lam1, A.lam2);
        const T* lprev = pick(S.ip, A.lam0, A.lam1, A.lam2);
        T* lnew = pick(S.in_, A.lam0, A.lam1, A.lam2);
        const V4<T>* uY = pick4(S.jY, A.u0, A.u1, A.u2, A.u3);
        {
            double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            // ---- contact pass: g = dt^2 n.(u_i(y) - u_j(y)) + c, l+ = P(y - alpha g)
            const int ntrip = (int)ntrip_c;
            auto issue_lam = [&](int k) {
                const int sl = (k % GC) * NT + tid;
                const long long c = base + (long long)k * S_;
                const bool on = k < ntrip && c < C;
                const long long cc = on ? c : 0;
                cp_val(s_l + sl, lam + cc, on);
                cp_val(s_lp + sl, lprev + cc, on && use_prev);
            };
            auto issue = [&](int k) {
                issue_geom(k);
                issue_lam(k);
                cp_commit();
            };
            // u(y) of the contact's two bodies (written by other blocks; see the comment at the kernel)
            auto gather = [&](int k, T* g) {
                const int sl = (k % GC) * NT + tid;
                const int2 ij = s_ij[sl];
                const bool on = k < ntrip && base + (long long)k * S_ < C;
                V4<T> ui, uj;
                ui.x = ui.y = ui.z = uj.x = uj.y = uj.z = (T)0;
                if (on && ij.x >= A.nin) ui = ld4(uY + (ij.x - A.nin));
                if (on && ij.y >= A.nin) uj = ld4(uY + (ij.y - A.nin));
                g[0] = ui.x; g[1] = ui.y; g[2] = ui.z;
                g[3] = uj.x; g[4] = uj.y; g[5] = uj.z;
            };
            // prologue: the geometry of stages 0..GC-2 in one group (issued before the
            // last barrier when geom_issued), then their multipliers one group per stage
            if (!geom_issued)
#pragma unroll 1
                for (int k = 0; k < GC - 1; ++k) issue_geom(k);
            cp_commit();
            geom_issued = false;
#pragma unroll 1
            for (int k = 0; k < GC - 1; ++k) {
                issue_lam(k);
                cp_commit();
            }
            cp_wait<GC - 2>();
            // trip k: commit stage k + GC - 1, wait for stage k + GD, gather trip k + GD's
            // u(y), then compute trip k with the u(y) gathered GD trips ago.  Three register
            // sets in rotation (the loop unrolled by three) so that no gather is forced to
            // complete before its own trip.
            static_assert(GD == 2, "three gather sets in rotation");
            auto trip = [&](int k, const T* g, T* fill) {
                issue(k + GC - 1);
                cp_wait<GC - 1 - GD>();  // stages up to k + GD have landed
                gather(k + GD, fill);
                const long long c = base + (long long)k * S_;
                if (k < ntrip && c < C) {
                    const int sl = (k % GC) * NT + tid;
                    const V4<T> nc = s_nc[sl];
                    // bodies below nin (obstacles) gathered as zeros: same sum as skipping them
                    V4<T> ui, uj;
                    ui.x = g[0]; ui.y = g[1]; ui.z = g[2];
                    uj.x = g[3]; uj.y = g[4]; uj.z = g[5];
                    int sv = -1;
                    T l2 = 0, q2 = 0, lp2 = 0;
                    if (PROB == kViscous) {
                        sv = A.slot[c];
                        if (sv >= 0) {
                            l2 = lam[sv];
                            if (use_prev) q2 = lprev[sv];
                        }
                    }
                    contact_update<T, DIM, PROB>(A, c, nc, ui, uj, s_l[sl], s_lp[sl], sv, l2, q2, &lp2, lnew, beta,
                                                 use_prev, bt, alpha, s);
                }
            };
            T g0[6], g1[6], g2[6];
            gather(0, g0);
            gather(1, g1);
#pragma unroll 1
            for (int k = 0; k < ntrip; k += 3) {
                trip(k, g0, g2);
                trip(k + 1, g1, g0);
                trip(k + 2, g2, g1);
            }
            cp_wait<0>();
            // FP32 needs four of the sums (|d|^2, |l+ - l|^2, g.(l+ - l), |l+|^2)
            constexpr int NS = sizeof(T) == 4 ? 4 : 8;
            if (NS == 4) {
                s[0] = s[1];
                s[1] = s[4];
                s[2] = s[5];
                s[3] = s[6];
            }
            G.template publish<NS>(s, red);
            // every thread is past its contact loop: the particle pass's first stages fill
            // the shared memory while the sums travel (u(l) copied whatever beta is)
            {
                const V4<T>* uL0 = pick4(S.jL, A.u0, A.u1, A.u2, A.u3);
#pragma unroll 1
                for (int k = 0; k < GP - 1; ++k) issue_body(k, uL0, uY, true);
            }
            if (tid < 32) {
                const Momentum mo = prepare_momentum(S);
                double t[NS];
                const bool ok = G.template collect<NS>(t);
                if (tid == 0) {
                    if (!ok) {
                        S.err = 1;
                        S.done = 1;
                    }
                    decide_momentum<T>(S, t, bt, A.dynamic, mo);
                }
            }
            G.next();
        }
        __syncthreads();
        if (S.err) break;
        {
            // ---- particle pass: w = B^T l+, u = M^-1 w, u(next y)
            V4<T>* uL = pick4(S.jL, A.u0, A.u1, A.u2, A.u3);
            V4<T>* uN = pick4(S.jN, A.u0, A.u1, A.u2, A.u3);
            V4<T>* uYN = pick4(S.jYN, A.u0, A.u1, A.u2, A.u3);
            const T bn_ = (T)S.beta_n;
            double sw = 0.0, sq = 0.0;
            // one body per thread; its incidence records, then the l+ gathers they index,
            // are issued in batches so several loads are in flight per thread
            constexpr int KB = 4;
            const long long ntrip = ntrip_p;
            // stages 0..GP-2 were issued before the barrier
#pragma unroll 1
            for (long long kt = 0; kt < ntrip; ++kt) {
                issue_body(kt + GP - 1, uL, uY, bn_ != (T)0);
                cp_wait<GP - 1>();  // stage kt has landed
                const long long p = base + kt * S_;
                if (p >= A.na) continue;
                const int sl = (int)(kt % GP) * NT + tid;
                T w0 = 0, w1 = 0, w2 = 0;
                const int k0 = s_p0[sl], k1 = s_p1[sl] - k0;
                const IncWalk wk = inc_walk(lay, sizeof(T) / 4, p, k0);
                for (int kb = 0; kb < k1; kb += KB) {
                    T ex[KB], ey[KB], ez[KB], mu[KB];
                    int ci[KB];
#pragma unroll
                    for (int q = 0; q < KB; ++q) {
                        ex[q] = ey[q] = ez[q] = mu[q] = (T)0;
                        ci[q] = -1;
                        if (kb + q < k1) {
                            const V4<T> e = PAST_L2 ? ld_inch(A.inc, wk, kb + q, pol) : ld_inc(A.inc, wk, kb + q);
                            ex[q] = e.x;
                            ey[q] = e.y;
                            ez[q] = e.z;
                            ci[q] = idx_of(e.w);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < KB; ++q)
                        if (ci[q] >= 0) {
                            mu[q] = lnew[ci[q]];
                            if (PROB == kViscous) {
                                const int sv = A.slot[ci[q]];
                                if (sv >= 0) mu[q] -= lnew[sv];
                            }
                        }
#pragma unroll
                    for (int q = 0; q < KB; ++q) {
                        w0 += mu[q] * ex[q];
                        w1 += mu[q] * ey[q];
                        if (DIM == 3) w2 += mu[q] * ez[q];
                    }
                }
                const T im = s_im[sl];
                const T n0 = im * w0, n1 = im * w1, n2 = im * w2;
                st4(uN + p, n0, n1, n2);
                // w.u gives F(l+) for the reference's test (FP64); FP32 tests the curvature
                if (sizeof(T) == 8) sw += (double)w0 * (double)n0 + (double)w1 * (double)n1 + (double)w2 * (double)n2;
                if (sizeof(T) == 4) {
                    // m |u(l+) - u(y)|^2: the curvature d^T Q d / dt^2 along d = l+ - y
                    const V4<T> uy = s_uy[sl];
                    const double d0 = (double)n0 - (double)uy.x, d1 = (double)n1 - (double)uy.y,
                                 d2 = (double)n2 - (double)uy.z;
                    sq += (d0 * d0 + d1 * d1 + d2 * d2) / (double)im;
                }
                if (bn_ != (T)0) {
                    const V4<T> ul = s_ul[sl];
                    st4(uYN + p, n0 + bn_ * (n0 - ul.x), n1 + bn_ * (n1 - ul.y), n2 + bn_ * (n2 - ul.z));
                } else {
                    st4(uYN + p, n0, n1, n2);
                }
            }
            cp_wait<0>();
            // FP64 reduces w.u, FP32 the curvature
            double sw1[1] = {sizeof(T) == 4 ? sq : sw};
            G.template publish<1>(sw1, red);
            // the next iteration's first contact geometry, while the sums travel
#pragma unroll 1
            for (int k = 0; k < GC - 1; ++k) issue_geom(k);
            geom_issued = true;
            if (tid < 32) {
                const NextStep ns = prepare_step<T>(S, A.tol);
                double t[1];
                const bool ok = G.template collect<1>(t);
                if (tid == 0) {
                    if (!ok) {
                        S.err = 1;
                        S.done = 1;
                    } else {
                        decide_step<T>(S, t[0], t[0], A.dt2, A.dynamic, A.max_ite, ns);
                    }
                }
            }
            G.next();
            __syncthreads();
            if (S.done) break;
        }
    }
    // copies issued for an iteration that did not run (wait_group does not cover
    // uncommitted copies: commit them first)
    cp_commit();
    cp_wait<0>();
    if (blockIdx.x == 0 && threadIdx.x == 0) write_result(A.result, S);
}

// ------------------------------------------------------------------ resident form
// Up to RC contacts and one body per thread of the grid: their records, multipliers and
// velocities stay with the thread for the whole solve, so a pass is its gathers (u(y) of a
// contact's bodies, l+ of a body's contacts) and little else.  In FP64 all of it is in registers;
// the 80 of FP32's 768 threads spill 32, 104 and 248 B a thread at one, two and four contacts
// (Viscous 68, 160 and 356 B) to the L1.  An iteration has one barrier
// between the passes and one exchange of sums after them: the particle pass forms u(next y)
// with the momentum of an accepted step, after a restart u(l+) itself is the next y.
// Solves of up to 16 blocks with one contact a thread run as ONE cluster (CL): its barriers and
// distributed shared memory take the place of 2 x ~5000 cycles of fences, stores and polls
// through L2 per iteration.  What bounds either form is that chain of latencies.
// Against the streaming form, microseconds per iteration: FP64 2k contacts 9.9 -> 4.7 (cluster),
// 20k 13.8 -> 11.4, 133k 13.9 -> 11.4 (two contacts a thread); FP32 61k 12.9 -> 10.6, 451k 16.0 -> 15.7
// (four a thread: the gathers' L2 traffic is the larger part there).
template <typename T, int DIM, int PROB, int RC, bool CL>
__global__ void __launch_bounds__(SphShape<T>::threads, 1) k_apgd_sph_res(SphArgs<T> A) {
    __shared__ ApgdState S;
    __shared__ double red[8][32];
    __shared__ Momentum s_mo;
    __shared__ NextStep s_ns;
    constexpr int KB = sizeof(T) == 4 ? 6 : 4;  // incidence records loaded while the barrier waits
    const int NT = blockDim.x, tid = threadIdx.x;
    const int C = A.sizes->C;
    const IncLayout lay = inc_layout(A.sizes, A.na, A.inc_slots);
    typename SyncOf<CL, true>::type G;
    sync_init(G, A.sums, A.bar, A.stall != 0 && blockIdx.x == 0);
    if (tid == 0) state_init(S, A.alpha);
    __syncthreads();
    if (A.curvature_start) curvature_step<T, DIM, PROB>(A, C, lay, S, G);
    const int base = (int)blockIdx.x * NT + tid, stride = (int)gridDim.x * NT;
    // this thread's contacts
    V4<T> nc[RC];
    int2 ij[RC];
    T lm[RC], lq[RC], ln[RC];
    int sv[PROB == kViscous ? RC : 1];
    T lm2[PROB == kViscous ? RC : 1], lq2[PROB == kViscous ? RC : 1], ln2[PROB == kViscous ? RC : 1];
#pragma unroll
    for (int r = 0; r < RC; ++r) {
        const int c = base + r * stride;
        ij[r] = make_int2(-1, -1);
        nc[r].x = nc[r].y = nc[r].z = nc[r].w = (T)0;
        lm[r] = lq[r] = ln[r] = (T)0;
        if (c < C) {
            nc[r] = ld4(A.nc + c);
            ij[r] = A.cij[c];
        }
        if (PROB == kViscous) {
            sv[r] = c < C ? A.slot[c] : -1;
            lm2[r] = lq2[r] = ln2[r] = (T)0;
        }
    }
    // this thread's body
    const bool body = base < A.na;
    const int k0 = body ? A.inc_ptr[base] : 0, cnt = body ? A.inc_ptr[base + 1] - k0 : 0;
    const IncWalk wk = inc_walk(lay, sizeof(T) / 4, base, k0);
    const T im = body ? A.invm[base] : (T)0;
    T ul0 = 0, ul1 = 0, ul2 = 0, uy0 = 0, uy1 = 0, uy2 = 0;
    for (;;) {
        if (S.done) break;
        const double alpha = S.alpha;
        const bool bt = S.bt != 0, use_prev = S.use_prev != 0;
        const T beta = (T)S.beta;
        T* lnew = pick(S.in_, A.lam0, A.lam1, A.lam2);
        const V4<T>* uY = pick4(S.jY, A.u0, A.u1, A.u2, A.u3);
        double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        // ---- contact pass
        {
            V4<T> gi[RC], gj[RC];
#pragma unroll
            for (int r = 0; r < RC; ++r) {
                gi[r].x = gi[r].y = gi[r].z = gj[r].x = gj[r].y = gj[r].z = (T)0;
                if (ij[r].x >= A.nin) gi[r] = ld4(uY + (ij[r].x - A.nin));
                if (ij[r].y >= A.nin) gj[r] = ld4(uY + (ij[r].y - A.nin));
            }
#pragma unroll
            for (int r = 0; r < RC; ++r) {
                if (ij[r].y < 0) continue;
                const int c = base + r * stride;
                const int e = PROB == kViscous ? r : 0;
                ln[r] = contact_update<T, DIM, PROB>(A, c, nc[r], gi[r], gj[r], lm[r], lq[r], PROB == kViscous ? sv[e] : -1,
                                                     lm2[e], lq2[e], &ln2[e], lnew, beta, use_prev, bt, alpha, s);
            }
        }
        G.arrive();
        // while the barrier waits: the warps' contact sums (FP32 reads |d|^2, |l+ - l|^2, g.(l+ - l) and
        // |l+|^2), what the decisions need, and the first incidence records
        if (sizeof(T) == 4) {
            s[0] = s[1];
            s[1] = s[4];
            s[2] = s[5];
            s[3] = s[6];
            s[4] = s[5] = s[6] = 0.0;
        }
        if (!CL) warp_sums<8>(s, red);
        if (tid == 32) s_mo = prepare_momentum(S);
        if (tid == 64) s_ns = prepare_step<T>(S, A.tol);
        V4<T> e[KB];
#pragma unroll
        for (int q = 0; q < KB; ++q)
            if (q < cnt) e[q] = ld_inc(A.inc, wk, q);
        if (!G.wait()) {
            if (tid == 0) {
                S.err = 1;
                S.done = 1;
            }
            break;
        }
        // the momentum was written after this block arrived: the cluster's wait does not order it
        // (the grid's wait ends in a block barrier)
        if (CL) __syncthreads();
        const T bn_ = (T)s_mo.beta;
        // ---- particle pass: w = B^T l+, u = M^-1 w, u(next y)
        V4<T>* uN = pick4(S.jN, A.u0, A.u1, A.u2, A.u3);
        V4<T>* uYN = pick4(S.jYN, A.u0, A.u1, A.u2, A.u3);
        T n0 = 0, n1 = 0, n2 = 0, y0 = 0, y1 = 0, y2 = 0;
        double sw = 0.0;
        if (body) {
            T w0 = 0, w1 = 0, w2 = 0;
            for (int kb = 0; kb < cnt; kb += KB) {
                T mu[KB];
                if (kb > 0)
#pragma unroll
                    for (int q = 0; q < KB; ++q)
                        if (kb + q < cnt) e[q] = ld_inc(A.inc, wk, kb + q);
#pragma unroll
                for (int q = 0; q < KB; ++q) {
                    mu[q] = (T)0;
                    if (kb + q < cnt) {
                        const int ci = idx_of(e[q].w);
                        mu[q] = lnew[ci];
                        if (PROB == kViscous) {
                            const int sl = A.slot[ci];
                            if (sl >= 0) mu[q] -= lnew[sl];
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < KB; ++q) {
                    if (kb + q >= cnt) continue;
                    w0 += mu[q] * e[q].x;
                    w1 += mu[q] * e[q].y;
                    if (DIM == 3) w2 += mu[q] * e[q].z;
                }
            }
            n0 = mul_rn(im, w0);
            n1 = mul_rn(im, w1);
            n2 = mul_rn(im, w2);
            st4(uN + base, n0, n1, n2);
            // w.u gives F(l+) for the reference's test (FP64); FP32 tests the curvature
            if (sizeof(T) == 8) {
                sw += (double)w0 * (double)n0 + (double)w1 * (double)n1 + (double)w2 * (double)n2;
            } else {
                const double d0 = (double)n0 - (double)uy0, d1 = (double)n1 - (double)uy1, d2 = (double)n2 - (double)uy2;
                sw += (d0 * d0 + d1 * d1 + d2 * d2) / (double)im;
            }
            y0 = n0;
            y1 = n1;
            y2 = n2;
            if (bn_ != (T)0) {
                y0 = fma_rn(bn_, add_rn(n0, -ul0), n0);
                y1 = fma_rn(bn_, add_rn(n1, -ul1), n1);
                y2 = fma_rn(bn_, add_rn(n2, -ul2), n2);
            }
            st4(uYN + base, y0, y1, y2);
        }
        // ---- the sums, the decisions
        if (CL) {
            s[sizeof(T) == 4 ? 4 : 7] = sw;
            warp_sums<8>(s, red);  // a cluster's barrier does not leave the time
        } else {
            warp_sum_to(sw, red[sizeof(T) == 4 ? 4 : 7]);
        }
        double t[8];
        const bool ok = G.template sums<8>(red, t);
        if (tid < 32) {
            // the two square roots side by side
            const double sq = sqrt(tid == 0 ? t[sizeof(T) == 4 ? 1 : 4] : t[3]);
            const double sq1 = __shfl_sync(0xffffffffu, sq, 1);
            if (tid == 0) {
                if (!ok) {
                    S.err = 1;
                    S.done = 1;
                } else {
                    decide_momentum<T>(S, t, bt, A.dynamic, s_mo);
                    const double last = t[sizeof(T) == 4 ? 4 : 7];
                    decide_step<T>(S, last, last, A.dt2, A.dynamic, A.max_ite, step_of<T>(s_ns, A.tol, sq, sq1));
                    if (!S.bt) reuse_buffers(S);
                }
            }
        }
        __syncthreads();
        if (!S.bt) {
#pragma unroll
            for (int r = 0; r < RC; ++r) {
                lq[r] = lm[r];
                lm[r] = ln[r];
                if (PROB == kViscous) {
                    lq2[r] = lm2[r];
                    lm2[r] = ln2[r];
                }
            }
            ul0 = n0;
            ul1 = n1;
            ul2 = n2;
            uy0 = S.restart ? n0 : y0;
            uy1 = S.restart ? n1 : y1;
            uy2 = S.restart ? n2 : y2;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) write_result(A.result, S);
    G.finish();
}

// ------------------------------------------------------------------ packing
__global__ void k_pack_cij(const int* ci, const int* cj, int2* cij, const Sizes* sizes) {
    GRID_STRIDE(c, sizes->C) { cij[c] = make_int2(ci[c], cj[c]); }
}
template <typename T>
__global__ void k_pack_nc(const double* bn, const double* cv, V4<T>* nc, const Sizes* sizes) {
    GRID_STRIDE(c, sizes->C) {
        V4<T> r;
        r.x = (T)bn[3 * c];
        r.y = (T)bn[3 * c + 1];
        r.z = (T)bn[3 * c + 2];
        r.w = (T)cv[c];
        nc[c] = r;
    }
}
template <typename T>
__device__ __forceinline__ T idx_bits(int c);
template <>
__device__ __forceinline__ float idx_bits<float>(int c) { return __int_as_float(c); }
template <>
__device__ __forceinline__ double idx_bits<double>(int c) { return __longlong_as_double((long long)c); }

template <typename T>
__device__ __forceinline__ void st_inc(Q16<T>* inc, long long at, int vs, double sg, const double* n, int c);
template <>
__device__ __forceinline__ void st_inc<float>(float4* inc, long long at, int, double sg, const double* n, int c) {
    inc[at] = make_float4((float)(sg * n[0]), (float)(sg * n[1]), (float)(sg * n[2]), idx_bits<float>(c));
}
template <>
__device__ __forceinline__ void st_inc<double>(double2* inc, long long at, int vs, double sg, const double* n, int c) {
    inc[at] = make_double2(sg * n[0], sg * n[1]);
    inc[at + vs] = make_double2(sg * n[2], idx_bits<double>(c));
}
// slots: the records `inc` holds; a list longer than that is cut (the no-allocation entry
// point rejects such lists before this runs; the engine sizes `inc` for every list)
template <typename T>
__global__ void k_pack_inc(int na, const int* ptr, const int* idx, const double* bn, Q16<T>* inc, long long slots,
                           const Sizes* sizes) {
    constexpr int nv = sizeof(T) / 4;
    const IncLayout lay = inc_layout(sizes, na, slots);
    if (lay.width) {
        const long long tot = (long long)lay.width * 32 * ((na + 31) / 32);
        GRID_STRIDE(t, tot) {
            const long long row = t >> 5, g = row / lay.width, p = g * 32 + (t & 31);
            const int r = (int)(row - g * lay.width);
            if (p >= na) continue;
            const int k0 = ptr[p];
            if (r >= ptr[p + 1] - k0) continue;
            const unsigned e = (unsigned)idx[k0 + r];
            const int c = (int)(e & 0x7fffffffu);
            st_inc<T>(inc, row * nv * 32 + (t & 31), 32, (e >> 31) ? -1.0 : 1.0, bn + 3 * (long long)c, c);
        }
        return;
    }
    const long long tot = ptr[na] < slots ? (long long)ptr[na] : slots;
    GRID_STRIDE(k, tot) {
        const unsigned e = (unsigned)idx[k];
        const int c = (int)(e & 0x7fffffffu);
        st_inc<T>(inc, k * nv, 1, (e >> 31) ? -1.0 : 1.0, bn + 3 * (long long)c, c);
    }
}

// ------------------------------------------------------------------ FP64 helpers (mixed form)
template <int DIM, int PROB>
__global__ void k_sph_particle64(int na, const int* ptr, const double2* inc, long long slots, const Sizes* sizes,
                                 const int* slot, const double* invm, const double* lam, dvec4* u) {
    const IncLayout lay = inc_layout(sizes, na, slots);
    GRID_STRIDE(p, na) {
        double w0 = 0, w1 = 0, w2 = 0;
        const int k0 = ptr[p], n = ptr[p + 1] - k0;
        const IncWalk wk = inc_walk(lay, 2, p, k0);
        for (int k = 0; k < n; ++k) {
            const dvec4 e = ld_inc(inc, wk, k);
            const int c = idx_of(e.w);
            double mu = lam[c];
            if (PROB == kViscous && slot[c] >= 0) mu -= lam[slot[c]];
            w0 += mu * e.x;
            w1 += mu * e.y;
            if (DIM == 3) w2 += mu * e.z;
        }
        const double im = invm[4 * (long long)p];
        st4(u + p, im * w0, im * w1, im * w2);
    }
}

template <int DIM, int PROB>
__global__ void k_sph_residual64(int nin, const int2* cij, const dvec4* nc, const int* slot, double dt2, const dvec4* u,
                                 double* g, unsigned long long* viol_bits, const Sizes* sizes) {
    double vmax = 0.0;
    GRID_STRIDE(c, sizes->C) {
        const int2 ij = cij[c];
        const dvec4 n = ld4(nc + c);
        double q = 0.0;
        if (ij.x >= nin) {
            const dvec4 a = ld4(u + (ij.x - nin));
            q += n.x * a.x + n.y * a.y + (DIM == 3 ? n.z * a.z : 0.0);
        }
        if (ij.y >= nin) {
            const dvec4 b = ld4(u + (ij.y - nin));
            q -= n.x * b.x + n.y * b.y + (DIM == 3 ? n.z * b.z : 0.0);
        }
        const double gg = dt2 * q + n.w;
        g[c] = gg;
        if (PROB == kViscous && slot[c] >= 0) g[slot[c]] = -gg;
        vmax = fmax(vmax, -gg);
    }
    if (vmax > 0.0) atomicMax(viol_bits, (unsigned long long)__double_as_longlong(vmax));
}

int blocks(long long n) {
    long long b = (n + 255) / 256;
    if (b < 1) b = 1;
    return (int)(b < 16 * kSMs ? b : 16 * kSMs);
}

// contacts a thread of the resident form can hold
template <typename T>
constexpr int kResidentContacts = sizeof(T) == 4 ? 4 : 2;

// Whether an iteration of the streaming form touches more than the L2 holds (126 MB, less what a
// solve that fits should leave to the rest).  FP32 only: 4.6M contacts 97.0 -> 91.7 us per iteration;
// in FP64 the multipliers and velocities alone are past it (154 us either way).
constexpr double kL2Bytes = 100.0 * (1 << 20);
template <typename T>
bool past_l2(double contacts, double bodies) {
    return sizeof(T) == 4 && contacts * (3 * sizeof(V4<T>) + sizeof(int2) + 3 * sizeof(T)) + bodies * 4 * sizeof(V4<T>) > kL2Bytes;
}

// the streaming form's shared memory
template <typename T, int DIM, int PROB>
void set_sph_smem() {
    static std::atomic<bool> done[kMaxDevices];
    once_per_device(done, [] {
        cudaFuncSetAttribute(k_apgd_sph<T, DIM, PROB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)SphOcc<T>::smem);
        if constexpr (sizeof(T) == 4)
            cudaFuncSetAttribute(k_apgd_sph<T, DIM, PROB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SphOcc<T>::smem);
    });
}

template <typename T, int DIM, int PROB>
int max_blocks_sph() {
    set_sph_smem<T, DIM, PROB>();
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_apgd_sph<T, DIM, PROB, false>, SphOcc<T>::threads,
                                                  SphOcc<T>::smem);
    int dev = 0, sms = kSMs;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::min(per_sm * sms, kSumMaxBlocks);
}

// the resident kernel as one cluster of n CTAs, where the device can hold one and takes the launch
template <typename T, int DIM, int PROB>
bool launch_cluster(SphArgs<T>& A, int n, cudaStream_t s) {
    static ClusterAble able;
    const int lg = log2_up(n);
    const auto kernel = k_apgd_sph_res<T, DIM, PROB, 1, true>;
    cudaLaunchAttribute attr[1];
    // blocks past the last contact and body only take part in the barriers
    const cudaLaunchConfig_t cfg = cluster_config(1 << lg, SphShape<T>::threads, s, attr);
    if (!cluster_fits(kernel, cfg, able, lg)) return false;
    if (cudaLaunchKernelEx(&cfg, kernel, A) != cudaSuccess) {
        cudaGetLastError();  // nothing ran: the caller takes the cooperative form
        return false;
    }
    g_sph_launches += 1;
    return true;
}

template <typename T, int DIM, int PROB, int RC>
cudaError_t launch_res(SphArgs<T>& A, int nblocks, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(SphShape<T>::threads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    g_sph_launches += 1;
    return cudaLaunchKernelEx(&cfg, k_apgd_sph_res<T, DIM, PROB, RC, false>, A);
}

// n_contacts: the host's count (the one in A.sizes)
template <typename T, int DIM, int PROB>
cudaError_t launch_t(SphArgs<T>& A, long long n_contacts, int nblocks, cudaStream_t s) {
    const long long threads = (long long)nblocks * SphShape<T>::threads;
    if (A.na <= threads && n_contacts <= kResidentContacts<T> * threads) {
        if (n_contacts <= threads) {
            // the wait-limit test needs the barrier that has a limit
            if (nblocks <= kMaxCluster && !A.stall && launch_cluster<T, DIM, PROB>(A, nblocks, s)) return cudaSuccess;
            return launch_res<T, DIM, PROB, 1>(A, nblocks, s);
        }
        if (n_contacts <= 2 * threads) return launch_res<T, DIM, PROB, 2>(A, nblocks, s);
        if constexpr (kResidentContacts<T> == 4) return launch_res<T, DIM, PROB, 4>(A, nblocks, s);
    }
    set_sph_smem<T, DIM, PROB>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(SphOcc<T>::threads);
    cfg.dynamicSmemBytes = SphOcc<T>::smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    g_sph_launches += 1;
    if constexpr (sizeof(T) == 4)
        if (past_l2<T>((double)n_contacts, (double)A.na))
            return cudaLaunchKernelEx(&cfg, k_apgd_sph<T, DIM, PROB, true>, A);
    return cudaLaunchKernelEx(&cfg, k_apgd_sph<T, DIM, PROB, false>, A);
}

}  // namespace

int apgd_sph_threads(bool fp32) { return fp32 ? SphOcc<float>::threads : SphOcc<double>::threads; }

int apgd_sph_max_blocks(int problem, int dim, bool fp32) {
#define MB(T, D, P) \
    if (dim == D && problem == P) return max_blocks_sph<T, D, P>();
    if (fp32) {
        MB(float, 2, 0) MB(float, 2, 2) MB(float, 3, 0) MB(float, 3, 2)
    } else {
        MB(double, 2, 0) MB(double, 2, 2) MB(double, 3, 0) MB(double, 3, 2)
    }
#undef MB
    return 0;
}

template <typename T>
cudaError_t launch_apgd_sph(int nin, int na, int dim, int problem, const ApgdSettings& st, SphSolve<T>& sb,
                            const Sizes* sizes, long long n_contacts, int nblocks, cudaStream_t s) {
    SphArgs<T> A;
    A.nin = nin;
    A.na = na;
    A.cij = sb.cij;
    A.nc = sb.nc;
    A.slot = sb.slot;
    A.shift = sb.shift;
    A.inc_ptr = sb.inc_ptr;
    A.inc = sb.inc;
    A.inc_slots = sb.inc_slots;
    A.invm = sb.invm;
    A.lam0 = sb.lam[0];
    A.lam1 = sb.lam[1];
    A.lam2 = sb.lam[2];
    A.u0 = sb.u[0];
    A.u1 = sb.u[1];
    A.u2 = sb.u[2];
    A.u3 = sb.u[3];
    A.sums = sb.sums;
    A.bar = sb.barrier;
    A.result = sb.result;
    A.sizes = sizes;
    A.alpha = st.alpha;
    A.tol = st.tol;
    A.dt2 = st.dt * st.dt;
    A.max_ite = st.max_ite;
    A.dynamic = st.dynamic;
    A.curvature_start = st.curvature_start;
    A.stall = st.stall;
#define LA(D, P) \
    if (dim == D && problem == P) return launch_t<T, D, P>(A, n_contacts, nblocks, s);
    LA(2, 0) LA(2, 2) LA(3, 0) LA(3, 2)
#undef LA
    return cudaErrorInvalidValue;
}
template cudaError_t launch_apgd_sph<double>(int, int, int, int, const ApgdSettings&, SphSolve<double>&, const Sizes*,
                                             long long, int, cudaStream_t);
template cudaError_t launch_apgd_sph<float>(int, int, int, int, const ApgdSettings&, SphSolve<float>&, const Sizes*,
                                            long long, int, cudaStream_t);

void launch_pack_cij(const int* ci, const int* cj, int2* cij, const Sizes* sizes, long long c_cap, cudaStream_t s) {
    k_pack_cij<<<blocks(c_cap), 256, 0, s>>>(ci, cj, cij, sizes);
    g_sph_launches += 1;
}
template <typename T>
void launch_pack_nc(const double* bn, const double* cvec, V4<T>* nc, const Sizes* sizes, long long c_cap,
                    cudaStream_t s) {
    k_pack_nc<T><<<blocks(c_cap), 256, 0, s>>>(bn, cvec, nc, sizes);
    g_sph_launches += 1;
}
template void launch_pack_nc<double>(const double*, const double*, dvec4*, const Sizes*, long long, cudaStream_t);
template void launch_pack_nc<float>(const double*, const double*, float4*, const Sizes*, long long, cudaStream_t);
template <typename T>
void launch_pack_inc(int na, const int* ptr, const int* idx, const double* bn, Q16<T>* inc, long long slots,
                     const Sizes* sizes, cudaStream_t s) {
    if (na <= 0) return;
    k_pack_inc<T><<<blocks(slots), 256, 0, s>>>(na, ptr, idx, bn, inc, slots, sizes);
    g_sph_launches += 1;
}
template void launch_pack_inc<double>(int, const int*, const int*, const double*, double2*, long long, const Sizes*,
                                      cudaStream_t);
template void launch_pack_inc<float>(int, const int*, const int*, const double*, float4*, long long, const Sizes*,
                                     cudaStream_t);

void launch_sph_particle64(int na, int dim, int problem, const int* ptr, const double2* inc, long long slots,
                           const Sizes* sizes, const int* slot, const double* invm, const double* lam, dvec4* u,
                           cudaStream_t s) {
    if (na <= 0) return;
#define PP(D, P) \
    if (dim == D && problem == P) k_sph_particle64<D, P><<<blocks(na), 256, 0, s>>>(na, ptr, inc, slots, sizes, slot, invm, lam, u);
    PP(2, 0) PP(2, 2) PP(3, 0) PP(3, 2)
#undef PP
    g_sph_launches += 1;
}

void launch_sph_residual64(int nin, int dim, int problem, const int2* cij, const dvec4* nc, const int* slot, double dt2,
                           const dvec4* u, double* g, unsigned long long* viol, const Sizes* sizes, long long c_cap,
                           cudaStream_t s) {
#define RR(D, P) \
    if (dim == D && problem == P) \
        k_sph_residual64<D, P><<<blocks(c_cap), 256, 0, s>>>(nin, cij, nc, slot, dt2, u, g, viol, sizes);
    RR(2, 0) RR(2, 2) RR(3, 0) RR(3, 2)
#undef RR
    g_sph_launches += 1;
}

// ------------------------------------------------------------------ entry point without allocation
//
// scopi_gpu_apgd_noalloc runs the FP64 torque-free APGD solve on caller-provided device
// arrays and keeps every intermediate array (packed contact and incidence records, the
// three multiplier buffers, the four per-body velocity buffers, block partials, the grid
// barrier and the result word) in g_noalloc_scratch below instead of cudaMalloc'd memory.
// Some callers cannot allocate device memory while they run the solve: a process whose
// device memory is owned by another allocator (a caching pool that has claimed the
// memory it will hand out), or a latency-critical loop where cudaMalloc / cudaFree would
// synchronise the device and stall the other streams.  They pass inputs and outputs only.
//
// The array is a file-scope __device__ variable, so every GPU that loads this library
// holds it (kNoAllocBytes, about 3.4 MB) until the process exits.  Its host-side name is
// only a stand-in for the device address, so at set-up the device address is fetched once
// per device with cudaGetSymbolAddress (with that device current) and passed to the
// kernels.  All calls share the array and it keeps the last call's contents: each call
// clears what must start at zero, and calls that overlap on the GPU (concurrent streams,
// or several host threads) race on it.
namespace {

constexpr long long kNoAllocMaxContacts = 16384;
constexpr long long kNoAllocMaxBodies = 8192;
static_assert(kNoAllocMaxContacts <= 32 * SphShape<double>::threads, "every size is resident, one contact a thread");

constexpr size_t kAlign = 256;
constexpr size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }
constexpr size_t kOffCij = 0;
constexpr size_t kOffNc = align_up(kOffCij + sizeof(int2) * kNoAllocMaxContacts);
constexpr size_t kOffInc = align_up(kOffNc + sizeof(dvec4) * kNoAllocMaxContacts);
constexpr size_t kOffInvm = align_up(kOffInc + sizeof(dvec4) * 2 * kNoAllocMaxContacts);
constexpr size_t kOffLam = align_up(kOffInvm + sizeof(double) * kNoAllocMaxBodies);
constexpr size_t kOffU = align_up(kOffLam + sizeof(double) * 3 * kNoAllocMaxContacts);
constexpr size_t kOffPart = align_up(kOffU + sizeof(dvec4) * 4 * kNoAllocMaxBodies);
constexpr size_t kOffBar = align_up(kOffPart + (size_t)kSumBytesPerBlock * apgdc::kSumMaxBlocks);
constexpr size_t kOffRes = align_up(kOffBar + 4 * sizeof(unsigned int));
constexpr size_t kOffSizes = align_up(kOffRes + sizeof(ApgdResult));
constexpr size_t kOffFlag = align_up(kOffSizes + sizeof(Sizes));
constexpr size_t kNoAllocBytes = align_up(kOffFlag + sizeof(unsigned int));

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

unsigned char* g_noalloc_dev[kMaxDevices] = {};
std::mutex g_noalloc_mutex;

// The solve's kernels on the current device: a size picks one of two (one cluster, or a grid with one
// contact a thread), and a kernel's code is loaded, into device memory, when it is first used.
// Loading both at the first call keeps a later call of another size from allocating.
template <int DIM>
cudaError_t noalloc_load() {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, k_apgd_sph_res<double, DIM, kNoFriction, 1, true>);
    return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_apgd_sph_res<double, DIM, kNoFriction, 1, false>);
}

// Device address of g_noalloc_scratch on the current device (set up on first use).
cudaError_t noalloc_scratch(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_dev[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e == cudaSuccess) e = noalloc_load<2>();
        if (e == cudaSuccess) e = noalloc_load<3>();
        if (e != cudaSuccess) return e;
        g_noalloc_dev[dev] = static_cast<unsigned char*>(ptr);
    }
    *out = g_noalloc_dev[dev];
    return cudaSuccess;
}

// The caller's contact list and incidence lists, checked before the solve reads them so that
// no index leaves its array: bit 1 inc_ptr does not start at 0 or decreases, bit 2
// inc_ptr[na] > 2 C (more records than the fixed array holds), bit 4 a record names a
// contact >= C, bit 8 a contact names a body outside [0, nb_inactive + n_active).
constexpr unsigned kBadPtr = 1u, kBadTotal = 2u, kBadRecord = 4u, kBadBody = 8u;
__global__ void k_noalloc_check(int na, int nbody, int C, const int* ci, const int* cj, const int* ptr, const int* idx,
                                unsigned* flag) {
    const int tot = ptr[na];
    const bool tot_ok = tot >= 0 && tot <= 2 * C;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (ptr[0] != 0) atomicOr(flag, kBadPtr);
        if (!tot_ok) atomicOr(flag, kBadTotal);
    }
    GRID_STRIDE(p, na) {
        if (ptr[p] > ptr[p + 1]) atomicOr(flag, kBadPtr);
    }
    if (tot_ok) GRID_STRIDE(k, tot) {
            if ((long long)((unsigned)idx[k] & 0x7fffffffu) >= (long long)C) atomicOr(flag, kBadRecord);
        }
    GRID_STRIDE(c, C) {
        const int a = ci[c], b = cj[c];
        if (a < 0 || a >= nbody || b < 0 || b >= nbody) atomicOr(flag, kBadBody);
    }
}

__global__ void k_noalloc_prepare(Sizes* sizes, int C, int na, const double* inv_mass, double* invm) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sizes->C = C;
        sizes->C_obs = 0;
        sizes->n_extra = 0;
        sizes->overflow = 0;
        sizes->inc_width = 0;  // rows one after the other: the fixed array has no room for columns
    }
    GRID_STRIDE(p, na) { invm[p] = inv_mass[p]; }
}

__global__ void k_noalloc_pack_nc(const double* normal, const double* cvec, dvec4* nc, int C) {
    GRID_STRIDE(c, C) { nc[c] = dvec4{normal[3 * c], normal[3 * c + 1], normal[3 * c + 2], cvec[c]}; }
}

// copy the result buffers chosen by the solve (recorded in *res) to the caller's outputs
__global__ void k_noalloc_output(const ApgdResult* res, const double* lam_base, const dvec4* u_base, int C, int na,
                                 double* lambda, double* u) {
    const double* lam = lam_base + (size_t)res->lam_buf * kNoAllocMaxContacts;
    const dvec4* ub = u_base + (size_t)res->u_buf * kNoAllocMaxBodies;
    GRID_STRIDE(k, C) { lambda[k] = lam[k]; }
    if (u)
        GRID_STRIDE(p, na) {
            const dvec4 v = ld4(ub + p);
            u[3 * p] = v.x;
            u[3 * p + 1] = v.y;
            u[3 * p + 2] = v.z;
        }
}

}  // namespace

void set_global_error(const char* msg);
void set_global_error2(const char* a, const char* b);

}  // namespace scopi_gpu

extern "C" int32_t scopi_gpu_apgd_noalloc(int32_t dim, int64_t n_active, int64_t nb_inactive, int64_t n_contacts,
                                          const int32_t* ci, const int32_t* cj, const double* normal,
                                          const double* c, const double* inv_mass, const int32_t* inc_ptr,
                                          const int32_t* inc_idx, double dt, double alpha, double tolerance,
                                          int64_t max_ite, int32_t dynamic_descent, double* lambda, double* u,
                                          int64_t* iterations, void* stream) {
    using namespace scopi_gpu;
    if (dim != 2 && dim != 3) {
        set_global_error("scopi_gpu_apgd_noalloc: dim must be 2 or 3");
        return SCOPI_GPU_EINVAL;
    }
    if (n_contacts < 0 || n_contacts > kNoAllocMaxContacts || n_active < 0 || n_active > kNoAllocMaxBodies ||
        nb_inactive < 0) {
        set_global_error("scopi_gpu_apgd_noalloc: size beyond the no-allocation limits (at most 16384 contacts and "
                         "8192 active bodies)");
        return SCOPI_GPU_EINVAL;
    }
    if (nb_inactive > 0x7fffffffLL - n_active) {
        set_global_error("scopi_gpu_apgd_noalloc: nb_inactive + n_active must fit in a 32-bit index");
        return SCOPI_GPU_EINVAL;
    }
    if (n_contacts > 0 && (!ci || !cj || !normal || !c || !inv_mass || !inc_ptr || !inc_idx || !lambda)) {
        set_global_error("scopi_gpu_apgd_noalloc: null array");
        return SCOPI_GPU_EINVAL;
    }
    if (!(alpha > 0) || max_ite < 1) {
        set_global_error("scopi_gpu_apgd_noalloc: alpha must be > 0 and max_ite >= 1");
        return SCOPI_GPU_EINVAL;
    }
    if (iterations) *iterations = 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_contacts == 0) {
        if (u && n_active > 0) {
            cudaError_t e = cudaMemsetAsync(u, 0, 3 * (size_t)n_active * sizeof(double), s);
            if (e != cudaSuccess) {
                set_global_error(cudaGetErrorString(e));
                return SCOPI_GPU_ECUDA;
            }
        }
        return SCOPI_GPU_OK;
    }
    unsigned char* base = nullptr;
    cudaError_t e = noalloc_scratch(&base);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: set-up: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    const int C = (int)n_contacts, na = (int)n_active;
    int2* cij = reinterpret_cast<int2*>(base + kOffCij);
    dvec4* nc = reinterpret_cast<dvec4*>(base + kOffNc);
    double2* inc = reinterpret_cast<double2*>(base + kOffInc);
    double* invm = reinterpret_cast<double*>(base + kOffInvm);
    double* lam = reinterpret_cast<double*>(base + kOffLam);
    dvec4* ub = reinterpret_cast<dvec4*>(base + kOffU);
    double* part = reinterpret_cast<double*>(base + kOffPart);
    unsigned int* bar = reinterpret_cast<unsigned int*>(base + kOffBar);
    ApgdResult* res = reinterpret_cast<ApgdResult*>(base + kOffRes);
    Sizes* sizes = reinterpret_cast<Sizes*>(base + kOffSizes);
    unsigned* flag = reinterpret_cast<unsigned*>(base + kOffFlag);
    // the caller's lists are checked first (one read-back): nothing below indexes with them
    // before they are known to stay inside their arrays
    e = cudaMemsetAsync(flag, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: cudaMemsetAsync: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    k_noalloc_check<<<blocks(std::max(C, na + 1)), 256, 0, s>>>(na, (int)(nb_inactive + n_active), C, ci, cj,
                                                                inc_ptr, inc_idx, flag);
    unsigned host_flag = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host_flag, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: input check: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    if (host_flag) {
        set_global_error((host_flag & kBadTotal)
                             ? "scopi_gpu_apgd_noalloc: inc_ptr[n_active] exceeds 2 * n_contacts"
                             : (host_flag & kBadPtr)
                                   ? "scopi_gpu_apgd_noalloc: inc_ptr must start at 0 and never decrease"
                                   : (host_flag & kBadRecord)
                                         ? "scopi_gpu_apgd_noalloc: inc_idx names a contact >= n_contacts"
                                         : "scopi_gpu_apgd_noalloc: ci/cj must be < nb_inactive + n_active");
        return SCOPI_GPU_EINVAL;
    }
    // the array keeps the previous call's contents: clear what the solve reads before writing
    // (lambda and lambda_prev, u(lambda), u(y), the barrier words, the result)
    struct Clear {
        void* p;
        size_t n;
    } clears[] = {{lam, 2 * sizeof(double) * kNoAllocMaxContacts},
                  {ub, sizeof(dvec4) * kNoAllocMaxBodies},
                  {ub + 2 * kNoAllocMaxBodies, sizeof(dvec4) * kNoAllocMaxBodies},
                  {bar, 4 * sizeof(unsigned int)},
                  {res, sizeof(ApgdResult)}};
    for (const Clear& cl : clears) {
        e = cudaMemsetAsync(cl.p, 0, cl.n, s);
        if (e != cudaSuccess) {
            set_global_error2("scopi_gpu_apgd_noalloc: cudaMemsetAsync: ", cudaGetErrorString(e));
            return SCOPI_GPU_ECUDA;
        }
    }
    k_noalloc_prepare<<<blocks(na), 256, 0, s>>>(sizes, C, na, inv_mass, invm);
    launch_pack_cij(ci, cj, cij, sizes, C, s);
    k_noalloc_pack_nc<<<blocks(C), 256, 0, s>>>(normal, c, nc, C);
    launch_pack_inc<double>(na, inc_ptr, inc_idx, normal, inc, 2 * (long long)C, sizes, s);
    SphArgs<double> A;
    A.nin = (int)nb_inactive;
    A.na = na;
    A.cij = cij;
    A.nc = nc;
    A.slot = nullptr;
    A.shift = nullptr;
    A.inc_ptr = inc_ptr;
    A.inc = inc;
    A.inc_slots = 2 * (long long)C;
    A.invm = invm;
    A.lam0 = lam;
    A.lam1 = lam + kNoAllocMaxContacts;
    A.lam2 = lam + 2 * kNoAllocMaxContacts;
    A.u0 = ub;
    A.u1 = ub + kNoAllocMaxBodies;
    A.u2 = ub + 2 * kNoAllocMaxBodies;
    A.u3 = ub + 3 * kNoAllocMaxBodies;
    A.sums = part;
    A.bar = bar;
    A.result = res;
    A.sizes = sizes;
    A.alpha = alpha;
    A.tol = tolerance;
    A.dt2 = dt * dt;
    A.max_ite = max_ite;
    A.dynamic = dynamic_descent ? 1 : 0;
    A.curvature_start = 0;
    A.stall = 0;
    int maxb = apgd_sph_max_blocks(kNoFriction, dim, false);
    const int thr = SphOcc<double>::threads;
    long long nb = (std::max<long long>(C, na) + thr - 1) / thr;
    if (nb < 1) nb = 1;
    if (nb > maxb) nb = maxb;
    e = cudaMemsetAsync(part, 0xff, (size_t)kSumBytesPerBlock * nb, s);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: cudaMemsetAsync: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    e = dim == 3 ? launch_t<double, 3, kNoFriction>(A, C, (int)nb, s)
                 : launch_t<double, 2, kNoFriction>(A, C, (int)nb, s);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: launch: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    k_noalloc_output<<<blocks(std::max(C, na)), 256, 0, s>>>(res, lam, ub, C, na, lambda, u);
    ApgdResult host_res;
    e = cudaMemcpyAsync(&host_res, res, sizeof(ApgdResult), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_global_error2("scopi_gpu_apgd_noalloc: ", cudaGetErrorString(e));
        return SCOPI_GPU_ECUDA;
    }
    if (iterations) *iterations = host_res.iterations;
    if (host_res.error) {
        set_global_error("scopi_gpu_apgd_noalloc: APGD grid barrier timed out");
        return SCOPI_GPU_ETIMEOUT;
    }
    return host_res.converged ? SCOPI_GPU_OK : SCOPI_GPU_ENOCONV;
}

