// apgd_fric.cu -- persistent APGD for the Friction problem (three multipliers per contact on
// the friction cone, 6-dof bodies), FrictionFixedPoint's solves included.  Same iteration,
// branch logic and stopping rule as apgd::operator() of include/scopi/solvers/apgd.hpp:148-221
// with LagrangeMultiplier<Friction> (lagrange_multiplier.hpp:208-273):
//     (A u)_c = v_i + P_i^T w_i - v_j - P_j^T w_j,   P = R^T [r]x,
// in two passes per iteration, each ended by grid sums (apgd_common.cuh):
//   contact pass : g = dt^2 A u(y) + c, l+ = P_K(y - alpha g);
//   particle pass: w = A^T l+, u = M^-1 w, and u(next y) = u + beta (u - u(l)), which the next
//                  contact pass gathers instead of two velocities.
// What bounds it: the latency of dependent gathers, then the bytes of the rows (24 values per
// contact, 10 per incidence in 3D).  The rows are therefore laid out for 16-byte coalesced
// loads: per contact in planes (vector v of contact c at [v][c]), per incidence in the order
// the particle pass walks them, with the incidence's sign already in P.  In 2D only what a
// planar rotation touches is stored (8 and 3 values).  Against the generic 6-dof kernel that
// served this problem before (rows and gathers in 4- and 8-byte loads, two gathers per body,
// 148 blocks of 256 threads, counter barriers), microseconds per iteration: 3D FP32 679k contacts
// 164 -> 66, FP64 44k 34.2 -> 18.3; 2D FP64 1.7k 22.9 -> 9.3.  The iterates are the same bits.
// The gathers are plain loads (the acquire of the barrier before a pass empties the L1, so they
// are fresh): against L2-only loads FP32 679k 65.7 -> 56.2, FP64 44k 16.1 -> 15.3.
// One barrier and one exchange of sums an iteration (instead of two exchanges), small solves in one
// cluster: FP32 679k 56.2 -> 49.3, 3k 9.4 -> 8.8; FP64 2D 1.7k 8.2 -> 5.4, 39k 10.8 -> 9.6; FP64 3D
// 118 contacts 9.9 -> 7.5, 44k 15.3 -> 15.5, 133k 19.8 -> 21.2 (there the registers are full).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>

#include "apgd_common.cuh"

namespace scopi_gpu {

static long long g_fric_launches = 0;
long long apgd_fric_launches() { return g_fric_launches; }

namespace {
using namespace apgdc;

template <typename T>
using Q4 = Q16<T>;

// values per contact row and per incidence record, and their 16-byte vectors.  Contact 3D:
// P_i (9), P_j (9), n, c; 2D: P_i[6..7], P_j[6..7], n, c.  Incidence 3D: +-P (9), index (, pad);
// 2D: +-P[6..7], pad, index.  index: contact, bit 31 = the body is the contact's j.
template <typename T, int DIM>
struct FricShape {
    static constexpr int per = 16 / sizeof(T);
    static constexpr int row = DIM == 3 ? 24 : 8;
    static constexpr int nv = row / per;
    static constexpr int inc = DIM == 3 ? (sizeof(T) == 4 ? 12 : 10) : 4;
    static constexpr int ni = inc / per;
    static constexpr int at_n = DIM == 3 ? 18 : 4, at_c = DIM == 3 ? 21 : 6, at_idx = DIM == 3 ? 9 : 3;
    static constexpr int nu = DIM == 3 ? 2 : 1;  // V4<T> per body of u: (v, 0), (w, 0); 2D (v, w, 0)
    static constexpr int dof = DIM == 3 ? 6 : 3;
};

// multipliers of a contact: three values in 3D (padded to a vector), two in 2D
template <typename T, int DIM>
struct Lam_of {
    using type = V4<T>;
};
template <>
struct Lam_of<float, 2> {
    using type = float2;
};
template <>
struct Lam_of<double, 2> {
    using type = double2;
};
template <typename T, int DIM>
using Lam = typename Lam_of<T, DIM>::type;

__device__ __forceinline__ void put4(float* o, const float4& v) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void put4(double* o, const double2& v) { o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void fld4(const float4* p, float* o) { put4(o, *p); }
__device__ __forceinline__ void fld4(const dvec4* p, double* o) {
    const double2* q = reinterpret_cast<const double2*>(p);
    put4(o, q[0]);
    put4(o + 2, q[1]);
}
__device__ __forceinline__ void fld4cg(const dvec4* p, double* o) {
    const double2* q = reinterpret_cast<const double2*>(p);
    put4(o, __ldcg(q));
    put4(o + 2, __ldcg(q + 1));
}
__device__ __forceinline__ void fst4(float4* p, const float* v) { *p = make_float4(v[0], v[1], v[2], 0.f); }
__device__ __forceinline__ void fst4(dvec4* p, const double* v) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0] = make_double2(v[0], v[1]);
    q[1] = make_double2(v[2], 0.0);
}
__device__ __forceinline__ void fld4(const float2* p, float* o) { const float2 v = *p; o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void fld4(const double2* p, double* o) { put4(o, *p); }
__device__ __forceinline__ void fld4cg(const double2* p, double* o) { put4(o, __ldcg(p)); }
__device__ __forceinline__ void fst4(float2* p, const float* v) { *p = make_float2(v[0], v[1]); }
__device__ __forceinline__ void fst4(double2* p, const double* v) { *p = make_double2(v[0], v[1]); }
__device__ __forceinline__ unsigned fidx(float w) { return (unsigned)__float_as_int(w); }
__device__ __forceinline__ unsigned fidx(double w) { return (unsigned)__double_as_longlong(w); }
template <typename T>
__device__ __forceinline__ T fidx_bits(unsigned e);
template <>
__device__ __forceinline__ float fidx_bits<float>(unsigned e) { return __int_as_float((int)e); }
template <>
__device__ __forceinline__ double fidx_bits<double>(unsigned e) { return __longlong_as_double((long long)e); }

template <typename T>
struct FricArgs {
    int nin, na;
    long long cap;         // plane stride of rec
    const int2* cij;
    const Q4<T>* rec;
    const double* shift;   // correction solves: 3 per contact (null = none)
    const int* inc_ptr;
    const Q4<T>* inc;      // IncLayout
    long long inc_slots;
    const V4<T>* invm;     // 1/m, 1/Jx, 1/Jy, 1/Jz (2D: 1/m, 0, 0, 1/Jz)
    void* lam[3];          // Lam<T, DIM> per contact
    V4<T>* u0;
    V4<T>* u1;
    V4<T>* u2;
    V4<T>* u3;
    void* qv;              // batches: dt^2 A u(y), Lam<T, DIM> per contact
    double* wu;            // batches: w.u per body
    T* lam_out;            // 3 per contact
    T* u_out;              // 6 per body (null: not wanted)
    double* sums;
    unsigned int* bar;
    ApgdResult* result;
    const Sizes* sizes;
    double alpha, tol, dt2, mu;
    long long max_ite;
    int dynamic, curvature_start, stall;
};

template <typename T, int DIM>
__device__ __forceinline__ Lam<T, DIM>* pick_lam(const FricArgs<T>& A, int k) {
    return static_cast<Lam<T, DIM>*>(k == 0 ? A.lam[0] : (k == 1 ? A.lam[1] : A.lam[2]));
}
template <typename T>
__device__ __forceinline__ V4<T>* pick_u(const FricArgs<T>& A, int k) {
    return k == 0 ? A.u0 : (k == 1 ? A.u1 : (k == 2 ? A.u2 : A.u3));
}

template <typename T, int DIM>
__device__ __forceinline__ void load_row(const Q4<T>* rec, long long cap, long long c, T* r) {
    using F = FricShape<T, DIM>;
#pragma unroll
    for (int v = 0; v < F::nv; ++v) put4(r + v * F::per, rec[v * cap + c]);
}
// the linear term of contact c alone
template <typename T, int DIM>
__device__ __forceinline__ void load_c(const Q4<T>* rec, long long cap, long long c, T* o) {
    using F = FricShape<T, DIM>;
    const T* r = reinterpret_cast<const T*>(rec);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const int e = F::at_c + d;
        o[d] = r[((e / F::per) * cap + c) * F::per + e % F::per];
    }
}
// u of a body: (v, w), 2D (vx, vy, w)
template <typename T, int DIM>
__device__ __forceinline__ void load_u(const V4<T>* u, long long p, T* o) {
    T t[4];
    fld4(u + p * FricShape<T, DIM>::nu, t);
    o[0] = t[0];
    o[1] = t[1];
    o[2] = t[2];
    if (DIM == 3) {
        fld4(u + 2 * p + 1, t);
        o[3] = t[0];
        o[4] = t[1];
        o[5] = t[2];
    }
}
template <typename T, int DIM>
__device__ __forceinline__ void store_u(V4<T>* u, long long p, const T* o) {
    fst4(u + p * FricShape<T, DIM>::nu, o);
    if (DIM == 3) fst4(u + 2 * p + 1, o + 3);
}

// v + P^T w of one body at the contact
template <typename T, int DIM>
__device__ __forceinline__ void point_velocity(const T* P, const T* u, T* o) {
    if (DIM == 3) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const T pt = fma_rn(P[6 + d], u[5], fma_rn(P[d], u[3], mul_rn(P[3 + d], u[4])));
            o[d] = add_rn(u[d], pt);
        }
    } else {
#pragma unroll
        for (int d = 0; d < 2; ++d) o[d] = add_rn(u[d], mul_rn(P[d], u[2]));
    }
}

// One contact of the contact pass: its row r, u(y) of its bodies, l and l_prev; writes l+ and
// adds its terms to s (FP64 g.d, |d|^2, c.l+, F(y), |l+ - l|^2, g.(l+ - l), |l+|^2; FP32
// |d|^2, |l+ - l|^2, g.(l+ - l), |l+|^2).
// SUMS false: s is left alone and dt^2 A u(y) goes to qout.
template <typename T, int DIM, bool SUMS = true>
__device__ __forceinline__ void contact_row(const T* r, const T* ui, const T* uj, const T* lam, const T* lprev,
                                            T beta, bool use_prev, bool bt, double alpha, double mu, T dt2,
                                            const double* shift, T* lout, double* s, T* qout = nullptr) {
    using F = FricShape<T, DIM>;
    T a[DIM], b[DIM];
    point_velocity<T, DIM>(r, ui, a);
    point_velocity<T, DIM>(r + (DIM == 3 ? 9 : 2), uj, b);
    double y[3], gm[3], z[3], n[3];
    T qy[DIM];
    n[2] = z[2] = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        qy[d] = mul_rn(add_rn(a[d], -b[d]), dt2);
        const T gg = add_rn(qy[d], r[F::at_c + d]);
        gm[d] = (double)gg;
        y[d] = use_prev ? (double)fma_rn(beta, add_rn(lam[d], -lprev[d]), lam[d]) : (double)lam[d];
        n[d] = (double)r[F::at_n + d];
        z[d] = fma_rn(-alpha, gm[d], y[d]);
        if (shift) z[d] += shift[d];
    }
    cone_project<DIM>(z, n, mu);
    constexpr bool f32 = sizeof(T) == 4;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const T lp = (T)(shift ? z[d] - shift[d] : z[d]);
        lout[d] = lp;
        if (!SUMS) {
            qout[d] = qy[d];
            continue;
        }
        const double dly = (double)lp - y[d], dll = (double)lp - (double)lam[d];
        if (!f32) {
            const double cc = (double)r[F::at_c + d];
            s[0] += gm[d] * dly;
            s[2] += cc * (double)lp;
            if (!bt) s[3] += y[d] * (0.5 * (double)qy[d] + cc);
        }
        s[f32 ? 0 : 1] += dly * dly;
        s[f32 ? 1 : 4] += dll * dll;
        s[f32 ? 2 : 5] += gm[d] * dll;
        s[f32 ? 3 : 6] += (double)lp * (double)lp;
    }
    if (DIM == 2) lout[2] = (T)0;
    if (DIM == 2 && !SUMS) qout[2] = (T)0;
}

// Incidence records [kb, kb + KB) of a body with n of them.
template <typename T, int DIM, int KB>
__device__ __forceinline__ void load_incs(const Q4<T>* inc, const IncWalk& wk, int kb, int n,
                                          T (&e)[KB][FricShape<T, DIM>::inc]) {
    using F = FricShape<T, DIM>;
#pragma unroll
    for (int q = 0; q < KB; ++q)
        if (kb + q < n)
#pragma unroll
            for (int v = 0; v < F::ni; ++v)
                put4(e[q] + v * F::per, inc[wk.first + (long long)(kb + q) * wk.rs + v * wk.vs]);
}
// w = A^T l+ of one body over its n incidences, KB records and multipliers in flight; e holds the
// first KB records
template <typename T, int DIM, int KB>
__device__ __forceinline__ void body_force(const Q4<T>* inc, const IncWalk& wk, const Lam<T, DIM>* lnew, int n, T* w,
                                           T (&e)[KB][FricShape<T, DIM>::inc]) {
    using F = FricShape<T, DIM>;
#pragma unroll
    for (int d = 0; d < F::dof; ++d) w[d] = (T)0;
    for (int kb = 0; kb < n; kb += KB) {
        T l[KB][4];
        if (kb > 0) load_incs<T, DIM, KB>(inc, wk, kb, n, e);
#pragma unroll
        for (int q = 0; q < KB; ++q)
            if (kb + q < n) fld4(lnew + (fidx(e[q][F::at_idx]) & 0x7fffffffu), l[q]);
#pragma unroll
        for (int q = 0; q < KB; ++q) {
            if (kb + q >= n) continue;
            const T* P = e[q];
            const T* f = l[q];
            const bool neg = (fidx(e[q][F::at_idx]) >> 31) != 0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) w[d] += neg ? -f[d] : f[d];
            if (DIM == 3) {
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    w[3 + d] = add_rn(w[3 + d], fma_rn(P[3 * d + 2], f[2], fma_rn(P[3 * d], f[0], mul_rn(P[3 * d + 1], f[1]))));
            } else {
                w[2] = add_rn(w[2], fma_rn(P[0], f[0], mul_rn(P[1], f[1])));
            }
        }
    }
}
template <typename T, int DIM, int KB>
__device__ __forceinline__ void body_force(const Q4<T>* inc, const IncWalk& wk, const Lam<T, DIM>* lnew, int n, T* w) {
    T e[KB][FricShape<T, DIM>::inc];
    load_incs<T, DIM, KB>(inc, wk, 0, n, e);
    body_force<T, DIM, KB>(inc, wk, lnew, n, w, e);
}
template <typename T, int DIM>
__device__ __forceinline__ void body_velocity(const T* im, const T* w, T* u) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) u[d] = im[0] * w[d];
    if (DIM == 3) {
        u[3] = im[1] * w[3];
        u[4] = im[2] * w[4];
        u[5] = im[3] * w[5];
    } else {
        u[2] = im[3] * w[2];
    }
}
// w.u
template <typename T, int DIM>
__device__ __forceinline__ double body_wu(const T* w, const T* u) {
    double acc = 0.0;
#pragma unroll
    for (int d = 0; d < FricShape<T, DIM>::dof; ++d) acc += (double)w[d] * (double)u[d];
    return acc;
}
// |u - uy|^2_M
template <typename T, int DIM>
__device__ __forceinline__ double body_curvature(const T* im, const T* u, const T* uy) {
    double q = 0.0;
#pragma unroll
    for (int d = 0; d < FricShape<T, DIM>::dof; ++d) {
        const T m = d < DIM ? im[0] : (DIM == 3 ? im[d - 2] : im[3]);
        const double dd = (double)u[d] - (double)uy[d];
        if (m > (T)0) q += dd * dd / (double)m;
    }
    return q;
}

constexpr long long kMaxBacktracks = 4000;

// Threads per block (one block per SM).  FP64 keeps the 256 threads whose per-thread sums its
// decisions have always been taken from; FP32 decisions do not hang on the last bits.
template <typename T>
struct FricThreads {
    static constexpr int value = sizeof(T) == 4 ? 512 : 256;
    static constexpr int kb = sizeof(T) == 4 ? 3 : 4;
};

template <typename T, int DIM, bool CL>
__global__ void __launch_bounds__(FricThreads<T>::value, 1) k_apgd_fric(FricArgs<T> A) {
    using F = FricShape<T, DIM>;
    constexpr int KB = FricThreads<T>::kb;
    __shared__ ApgdState S;
    __shared__ double red[8][32];
    __shared__ Momentum s_mo;
    __shared__ NextStep s_ns;
    const int tid = threadIdx.x;
    const int C = A.sizes->C;
    const IncLayout lay = inc_layout(A.sizes, A.na, A.inc_slots);
    typename SyncOf<CL, false>::type G;
    sync_init(G, A.sums, A.bar, A.stall != 0 && blockIdx.x == 0);
    if (tid == 0) state_init(S, A.alpha);
    __syncthreads();
    if (A.curvature_start) {
        // initial step from the curvature along the first projected-gradient direction d of the
        // cold start (in the candidate buffer, which the first contact pass overwrites), with
        // 256 threads per block: the sums set the step, so their order is kept in FP32 too
        const long long S0 = (long long)gridDim.x * 256, b0 = (long long)blockIdx.x * 256 + tid;
        Lam<T, DIM>* dbuf = pick_lam<T, DIM>(A, 2);
        double a[2] = {0.0, 0.0};
        if (tid < 256)
            for (long long c = b0; c < C; c += S0) {
                T r[F::row];
                load_row<T, DIM>(A.rec, A.cap, c, r);
                double z[3], n[3];
                n[2] = z[2] = 0.0;
                for (int d = 0; d < DIM; ++d) {
                    n[d] = (double)r[F::at_n + d];
                    z[d] = -(double)r[F::at_c + d] + (A.shift ? A.shift[3 * c + d] : 0.0);
                }
                cone_project<DIM>(z, n, A.mu);
                T v[3] = {(T)0, (T)0, (T)0};
                for (int d = 0; d < DIM; ++d) {
                    v[d] = (T)(z[d] - (A.shift ? A.shift[3 * c + d] : 0.0));
                    a[0] += (double)v[d] * (double)v[d];
                }
                fst4(dbuf + c, v);
            }
        double t1 = 0.0, t6 = 0.0;
        block_sum<2>(a);
        bool ok = G.exchange(a[0], t1);
        double b[2] = {0.0, 0.0};
        if (ok && tid < 256)
            for (long long p = b0; p < A.na; p += S0) {
                T w[F::dof], u[F::dof], im[4];
                const int k0 = A.inc_ptr[p];
                body_force<T, DIM, KB>(A.inc, inc_walk(lay, F::ni, p, k0), dbuf, A.inc_ptr[p + 1] - k0, w);
                fld4(A.invm + p, im);
                body_velocity<T, DIM>(im, w, u);
                b[0] += body_wu<T, DIM>(w, u);
            }
        block_sum<2>(b);
        if (ok) ok = G.exchange(b[0], t6);
        if (tid == 0) {
            double l;
            if (!ok) {
                S.err = 1;
                S.done = 1;
            } else if (initial_lipschitz(t1, t6, A.dt2, l)) {
                S.lipsch = l;
                S.alpha = 1.0 / l;
                S.lgood = l;
            }
        }
        __syncthreads();
    }
    const long long S_ = (long long)gridDim.x * blockDim.x, base = (long long)blockIdx.x * blockDim.x + tid;
    // of the first contact and (where there are registers for them) the first body, for the whole solve
    const int2 ij0 = base < C ? A.cij[base] : make_int2(0, 0);
    constexpr bool keep = sizeof(T) == 4 || CL;
    int kb0 = 0, n0 = 0;
    IncWalk wk0{};
    auto body0 = [&] {
        kb0 = base < A.na ? A.inc_ptr[base] : 0;
        n0 = base < A.na ? A.inc_ptr[base + 1] - kb0 : 0;
        wk0 = inc_walk(lay, F::ni, base, kb0);
    };
    if (keep) body0();
    for (;;) {
        if (S.done) break;
        const double alpha = S.alpha;
        const bool bt = S.bt != 0, use_prev = S.use_prev != 0;
        const T beta = (T)S.beta;
        const Lam<T, DIM>* lam = pick_lam<T, DIM>(A, S.il);
        const Lam<T, DIM>* lprev = pick_lam<T, DIM>(A, S.ip);
        Lam<T, DIM>* lnew = pick_lam<T, DIM>(A, S.in_);
        const V4<T>* uY = pick_u(A, S.jY);
        const V4<T>* uL = pick_u(A, S.jL);
        V4<T>* uN = pick_u(A, S.jN);
        V4<T>* uYN = pick_u(A, S.jYN);
        double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        // ---- contact pass
        {
            int2 ij = ij0;
#pragma unroll 1
            for (long long c = base; c < C; c += S_) {
                const int2 me = ij;
                if (c + S_ < C) ij = A.cij[c + S_];
                T ui[F::dof], uj[F::dof], r[F::row], lm[4], lq[4], lo[3];
#pragma unroll
                for (int d = 0; d < F::dof; ++d) ui[d] = uj[d] = (T)0;
                if (me.x >= A.nin) load_u<T, DIM>(uY, me.x - A.nin, ui);
                if (me.y >= A.nin) load_u<T, DIM>(uY, me.y - A.nin, uj);
                load_row<T, DIM>(A.rec, A.cap, c, r);
                fld4(lam + c, lm);
                if (use_prev) fld4(lprev + c, lq);
                contact_row<T, DIM>(r, ui, uj, lm, lq, beta, use_prev, bt, alpha, A.mu, (T)A.dt2,
                                    A.shift ? A.shift + 3 * c : nullptr, lo, s);
                fst4(lnew + c, lo);
            }
        }
        G.arrive();
        // while the barrier waits: the warps' contact sums, what the decisions need, and the first
        // incidence records
        if (!CL) warp_sums<8>(s, red);
        if (tid == 32) s_mo = prepare_momentum(S);
        if (tid == 64) s_ns = prepare_step<T>(S, A.tol);
        T e[KB][F::inc];
        if (!keep) body0();
        load_incs<T, DIM, KB>(A.inc, wk0, 0, n0, e);
        if (!G.wait()) {
            if (tid == 0) {
                S.err = 1;
                S.done = 1;
            }
            break;
        }
        if (CL) __syncthreads();  // the momentum was written after the arrival
        const T bn_ = (T)s_mo.beta;
        // ---- particle pass
        double sw = 0.0;
#pragma unroll 1
        for (long long p = base; p < A.na; p += S_) {
            T im[4], ul[F::dof], uy[F::dof], w[F::dof], u[F::dof];
            int n = n0;
            IncWalk wk = wk0;
            if (p != base) {
                const int kb = A.inc_ptr[p];
                n = A.inc_ptr[p + 1] - kb;
                wk = inc_walk(lay, F::ni, p, kb);
                load_incs<T, DIM, KB>(A.inc, wk, 0, n, e);
            }
            fld4(A.invm + p, im);
            if (bn_ != (T)0) load_u<T, DIM>(uL, p, ul);
            if (sizeof(T) == 4) load_u<T, DIM>(uY, p, uy);
            body_force<T, DIM, KB>(A.inc, wk, lnew, n, w, e);
            body_velocity<T, DIM>(im, w, u);
            store_u<T, DIM>(uN, p, u);
            // w.u gives F(l+) for the reference's test (FP64); FP32 tests the curvature
            if (sizeof(T) == 8)
                sw += body_wu<T, DIM>(w, u);
            else
                sw += body_curvature<T, DIM>(im, u, uy);
            if (bn_ != (T)0) {
#pragma unroll
                for (int d = 0; d < F::dof; ++d) u[d] = fma_rn(bn_, add_rn(u[d], -ul[d]), u[d]);
            }
            store_u<T, DIM>(uYN, p, u);
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
                    decide_step<T>(S, last, last, A.dt2, A.dynamic, A.max_ite, step_of<T>(s_ns, A.tol, sq, sq1),
                                   kMaxBacktracks);
                    if (!S.bt) reuse_buffers(S);
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    // the result, in the layouts of the other kernels (every thread its own contacts and bodies)
    const Lam<T, DIM>* lres = pick_lam<T, DIM>(A, S.il);
    const V4<T>* ures = pick_u(A, S.jL);
    for (long long c = base; c < C; c += S_) {
        T l[4];
        fld4(lres + c, l);
        for (int d = 0; d < 3; ++d) A.lam_out[3 * c + d] = d < DIM ? l[d] : (T)0;
    }
    if (A.u_out)
        for (long long p = base; p < A.na; p += S_) {
            T u[F::dof];
            load_u<T, DIM>(ures, p, u);
            T* o = A.u_out + 6 * p;
            if (DIM == 3) {
                for (int d = 0; d < 6; ++d) o[d] = u[d];
            } else {
                o[0] = u[0];
                o[1] = u[1];
                o[2] = o[3] = o[4] = (T)0;
                o[5] = u[2];
            }
        }
    if (blockIdx.x == 0 && tid == 0) write_result(A.result, S);
    G.finish();
}

// ------------------------------------------------------------------ batched scenes (FP64)
// One CTA per scene, or a cluster of CS CTAs for a large one (fric_batch_form): the same iteration on the scene's
// contacts (its obstacle rows [o0, o1), then its active rows [a0, a1)) and bodies [p0, p1), so
// every scene iterates until its own stopping test holds; the multipliers, the velocities and
// the scene's statistics with the violation max(0, -gap) of its final state go to fixed outputs.
//
// What bounds it: a scene's iteration is a chain of dependent FP64 work (square root and
// divisions of the cone projection, ~150 instructions a contact) on very few SMs.  The passes
// therefore run on all threads of the CTAs, whatever their number, and the sums are a pass of
// their own: the scene's decisions are taken from sums over 256 chains (chain t adds contacts
// t, t + 256, ... one after the other), whose bits do not depend on how the passes are split.
// A contact leaves dt^2 A u(y) behind for it, a body w.u; the multipliers are there anyway.
// The particle pass does not wait for the sums: it forms u(next y) with the momentum of an
// accepted step, and after a restart u(l+) itself is the next y.  96 2D scenes of 200 to 2000
// disks, milliseconds a step: the generic 6-dof rows on 256 threads 69.4; packed rows on 256
// threads with two contacts at a time 23.1; this form, clusters of two for the largest, 15.5.  Every
// split gives the same bits.
constexpr int kChains = 256;
template <int DIM>
constexpr int kBatchFricThreads = DIM == 2 ? 512 : 256;  // 128 registers hold a 2D row, 255 a 3D one

__device__ __forceinline__ void cluster_sync() {
    __syncwarp();  // an aligned barrier wants whole warps
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int CS>
__device__ __forceinline__ void scene_sync() {
    if (CS == 1)
        __syncthreads();
    else
        cluster_sync();
}

// Sums of a scene's chains: each warp's tree goes to every CTA of the scene (sh[value][warp of
// chains]); after scene_sync, warps in order.
struct SceneSums {
    double w[8][kChains / 32];  // contact sums
    double b[kChains / 32];     // w.u
    double vmax[8];             // one per CTA
    Momentum mo;                // of this iteration, and the steps after it
    NextStep next;
};
template <int CS>
__device__ __forceinline__ void share(double* at, double v) {
    if (CS == 1) {
        *at = v;
    } else {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        for (int r = 0; r < CS; ++r) *cl.map_shared_rank(at, r) = v;
    }
}

template <int DIM, int CS, int BT>
__device__ void fric_scene(const FricArgs<double>& A, const BatchFricScenes& B, int sc, int rank, ApgdState& S,
                           SceneSums& Q) {
    using T = double;
    using F = FricShape<T, DIM>;
    using L = Lam<T, DIM>;
    constexpr int NT = CS * BT;
    constexpr int VT = kChains / CS;           // chains of this CTA: [rank * VT, rank * VT + VT)
    constexpr int CT = BT < VT ? BT : VT;      // summed at a time
    constexpr int SPLIT = BT / VT >= 2 ? 2 : 1;  // threads per chain: the sums shared between two
    const int lt = threadIdx.x, tid = rank * BT + lt;
    const IncLayout lay = inc_layout(A.sizes, A.na, A.inc_slots);
    const int o0 = B.sc_o0[sc], n0 = B.sc_o1[sc] - o0, a0 = B.sc_a0[sc];
    const int nc = n0 + (B.sc_a1[sc] - a0);
    const int p0 = B.sc_p0[sc], p1 = B.sc_p1[sc];
    L* qv = static_cast<L*>(A.qv);
    auto contact_at = [&](int k) -> int { return k < n0 ? o0 + k : a0 + (k - n0); };
    if (lt == 0) {
        state_init(S, A.alpha);
        if (nc == 0) S.done = S.conv = 1;
    }
    // lambda = lambda_prev = 0 and u(lambda) = u(y) = 0 (cold start, apgd.hpp:152-159)
    const T zero[6] = {0, 0, 0, 0, 0, 0};
    for (int k = tid; k < nc; k += NT) {
        const int c = contact_at(k);
        fst4(pick_lam<T, DIM>(A, 0) + c, zero);
        fst4(pick_lam<T, DIM>(A, 1) + c, zero);
    }
    for (int p = p0 + tid; p < p1; p += NT) {
        store_u<T, DIM>(A.u0, p, zero);
        store_u<T, DIM>(A.u2, p, zero);
    }
    scene_sync<CS>();
    if (nc > 0 && A.curvature_start) {
        // L = 1.5 dt^2 |B^T d|^2_{M^-1} / |d|^2 along the first projected-gradient direction
        L* dbuf = pick_lam<T, DIM>(A, 2);
        for (int k = tid; k < nc; k += NT) {
            const int c = contact_at(k);
            T r[F::row];
            load_row<T, DIM>(A.rec, A.cap, c, r);
            double z[3], n[3];
            n[2] = z[2] = 0.0;
            for (int d = 0; d < DIM; ++d) {
                n[d] = r[F::at_n + d];
                z[d] = -r[F::at_c + d];
            }
            cone_project<DIM>(z, n, A.mu);
            fst4(dbuf + c, z);
        }
        scene_sync<CS>();
        for (int p = p0 + tid; p < p1; p += NT) {
            T w[F::dof], u[F::dof], im[4];
            const int k0 = A.inc_ptr[p];
            body_force<T, DIM, 3>(A.inc, inc_walk(lay, F::ni, p, k0), dbuf, A.inc_ptr[p + 1] - k0, w);
            fld4(A.invm + p, im);
            body_velocity<T, DIM>(im, w, u);
            A.wu[p] = body_wu<T, DIM>(w, u);
        }
        scene_sync<CS>();
        for (int q = lt; lt < CT && q < VT; q += CT) {
            double s[2] = {0.0, 0.0};
            const int vt = rank * VT + q;
            for (int k = vt; k < nc; k += kChains) {
                T z[4];
                fld4cg(dbuf + contact_at(k), z);
                for (int d = 0; d < DIM; ++d) s[0] += z[d] * z[d];
            }
            for (int p = p0 + vt; p < p1; p += kChains) s[1] += __ldcg(A.wu + p);
            const double x0 = multi_reduce<1>(s), x1 = multi_reduce<1>(s + 1);
            if ((lt & 31) == 0) {
                share<CS>(&Q.w[0][vt >> 5], x0);
                share<CS>(&Q.b[vt >> 5], x1);
            }
        }
        scene_sync<CS>();
        if (lt == 0) {
            double t0 = 0.0, t1 = 0.0, l;
            for (int w = 0; w < kChains / 32; ++w) t0 += Q.w[0][w];
            for (int w = 0; w < kChains / 32; ++w) t1 += Q.b[w];
            if (initial_lipschitz(t0, t1, A.dt2, l)) {
                S.lipsch = l;
                S.alpha = 1.0 / l;
                S.lgood = l;
            }
        }
    }
    __syncthreads();
    while (!S.done) {
        const double alpha = S.alpha;
        const bool bt = S.bt != 0, use_prev = S.use_prev != 0;
        const T beta = S.beta;
        const L* lam = pick_lam<T, DIM>(A, S.il);
        const L* lprev = pick_lam<T, DIM>(A, S.ip);
        L* lnew = pick_lam<T, DIM>(A, S.in_);
        const V4<T>* uY = pick_u(A, S.jY);
        const V4<T>* uL = pick_u(A, S.jL);
        V4<T>* uN = pick_u(A, S.jN);
        V4<T>* uYN = pick_u(A, S.jYN);
        // square roots and divisions that the decisions need, on two warps while the others begin
        if (lt == BT - 32) Q.mo = prepare_momentum(S);
        if (lt == BT - 64) Q.next = prepare_step<T>(S, A.tol);
        // ---- contact pass
#pragma unroll 1
        for (int k = tid; k < nc; k += NT) {
            const int c = contact_at(k);
            T ui[F::dof], uj[F::dof], r[F::row], lm[4], lq[4], lo[3], qo[3], s[8];
            const int2 ij = A.cij[c];
            load_row<T, DIM>(A.rec, A.cap, c, r);
            fld4(lam + c, lm);
            if (use_prev) fld4(lprev + c, lq);
#pragma unroll
            for (int d = 0; d < F::dof; ++d) ui[d] = uj[d] = (T)0;
            if (ij.x >= A.nin) load_u<T, DIM>(uY, ij.x - A.nin, ui);
            if (ij.y >= A.nin) load_u<T, DIM>(uY, ij.y - A.nin, uj);
            contact_row<T, DIM, false>(r, ui, uj, lm, lq, beta, use_prev, bt, alpha, A.mu, A.dt2, nullptr, lo, s, qo);
            fst4(lnew + c, lo);
            fst4(qv + c, qo);
        }
        scene_sync<CS>();
        // ---- the sums: chain vt, its first or second half of the values
        {
            constexpr int J = 2;  // contacts whose loads are in flight
            const int part = SPLIT == 2 ? lt / VT : 0;
#pragma unroll 1
            for (int q = lt - part * VT; lt < SPLIT * CT && q < VT; q += CT) {
                const int vt = rank * VT + q;
                double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
                for (int k = vt; k < nc; k += J * kChains) {
                    T lm[J][4], lq[J][4], lp[J][4], q[J][4], cc[J][4];
#pragma unroll
                    for (int e = 0; e < J; ++e) {
                        if (k + e * kChains >= nc) continue;
                        const int c = contact_at(k + e * kChains);
                        fld4cg(lam + c, lm[e]);
                        if (use_prev) fld4cg(lprev + c, lq[e]);
                        fld4cg(lnew + c, lp[e]);
                        fld4cg(qv + c, q[e]);
                        load_c<T, DIM>(A.rec, A.cap, c, cc[e]);
                    }
#pragma unroll
                    for (int e = 0; e < J; ++e) {
                        if (k + e * kChains >= nc) continue;
#pragma unroll
                        for (int d = 0; d < DIM; ++d) {
                            const double y =
                                use_prev ? fma_rn(beta, add_rn(lm[e][d], -lq[e][d]), lm[e][d]) : lm[e][d];
                            const double gm = add_rn(q[e][d], cc[e][d]), dly = add_rn(lp[e][d], -y),
                                         dll = add_rn(lp[e][d], -lm[e][d]);
                            if (SPLIT == 1 || part == 0) {
                                s[0] = fma_rn(gm, dly, s[0]);
                                s[1] = fma_rn(dly, dly, s[1]);
                                s[2] = fma_rn(cc[e][d], lp[e][d], s[2]);
                            }
                            if (SPLIT == 1 || part == 1) {
                                if (!bt) s[3] = fma_rn(y, fma_rn(0.5, q[e][d], cc[e][d]), s[3]);
                                s[4] = fma_rn(dll, dll, s[4]);
                                s[5] = fma_rn(gm, dll, s[5]);
                                s[6] = fma_rn(lp[e][d], lp[e][d], s[6]);
                            }
                        }
                    }
                }
                const double x = multi_reduce<8>(s);
                const int v = (lt & 31) >> 2;
                if ((lt & 3) == 0 && (SPLIT == 1 || (v >= 3) == (part == 1))) share<CS>(&Q.w[v][vt >> 5], x);
            }
        }
        // ---- particle pass
        const T bn_ = Q.mo.beta;
#pragma unroll 1
        for (int p = p0 + tid; p < p1; p += NT) {
            const int k0 = A.inc_ptr[p];
            T im[4], ul[F::dof], w[F::dof], u[F::dof];
            fld4(A.invm + p, im);
            if (bn_ != 0.0) load_u<T, DIM>(uL, p, ul);
            body_force<T, DIM, DIM == 2 ? 4 : 3>(A.inc, inc_walk(lay, F::ni, p, k0), lnew, A.inc_ptr[p + 1] - k0, w);
            body_velocity<T, DIM>(im, w, u);
            store_u<T, DIM>(uN, p, u);
            A.wu[p] = body_wu<T, DIM>(w, u);
            if (bn_ != 0.0) {
#pragma unroll
                for (int d = 0; d < F::dof; ++d) u[d] = fma_rn(bn_, add_rn(u[d], -ul[d]), u[d]);
            }
            store_u<T, DIM>(uYN, p, u);
        }
        scene_sync<CS>();
        // ---- w.u along the chains (every CTA all of them: one sum), then the decisions
        {
            for (int t = lt; t < kChains; t += BT) {
                double s[1] = {0.0};
                for (int p = p0 + t; p < p1; p += kChains) s[0] += __ldcg(A.wu + p);
                const double x = multi_reduce<1>(s);
                if ((t & 31) == 0) Q.b[t >> 5] = x;
            }
        }
        __syncthreads();
        if (lt < 32) {
            double x = 0.0;
            const double* row = lt < 7 ? Q.w[lt] : Q.b;
            if (lt < 8)
                for (int w = 0; w < kChains / 32; ++w) x += row[w];
            double t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = __shfl_sync(0xffffffffu, x, k);
            if (lt == 0) {
                decide_momentum<T>(S, t, bt, A.dynamic, Q.mo);
                NextStep ns = Q.next;
                ns.step = sqrt(S.last_step);
                decide_step<T>(S, t[7], 0.0, A.dt2, A.dynamic, A.max_ite, ns, kMaxBacktracks);
                if (!S.bt) reuse_buffers(S);
            }
        }
        __syncthreads();
    }
    // outputs and the violation max(0, -n.(dt^2 A u + C)) over the scene's contacts
    const L* lres = pick_lam<T, DIM>(A, S.il);
    const V4<T>* ures = pick_u(A, S.jL);
    double vmax = 0.0;
    for (int k = tid; k < nc; k += NT) {
        const int c = contact_at(k);
        const int2 ij = A.cij[c];
        T r[F::row], l[4], ui[F::dof], uj[F::dof], a[3], b[3];
        load_row<T, DIM>(A.rec, A.cap, c, r);
        fld4(lres + c, l);
        for (int d = 0; d < 3; ++d) A.lam_out[3 * (long long)c + d] = d < DIM ? l[d] : 0.0;
        for (int d = 0; d < F::dof; ++d) ui[d] = uj[d] = 0.0;
        if (ij.x >= A.nin) load_u<T, DIM>(ures, ij.x - A.nin, ui);
        if (ij.y >= A.nin) load_u<T, DIM>(ures, ij.y - A.nin, uj);
        point_velocity<T, DIM>(r, ui, a);
        point_velocity<T, DIM>(r + (DIM == 3 ? 9 : 2), uj, b);
        double gap = 0.0;
        for (int d = 0; d < DIM; ++d) gap += (A.dt2 * (a[d] - b[d]) + r[F::at_c + d]) * r[F::at_n + d];
        vmax = fmax(vmax, -gap);
    }
    for (int p = p0 + tid; p < p1; p += NT) {
        T u[F::dof];
        load_u<T, DIM>(ures, p, u);
        T* o = A.u_out + 6 * (long long)p;
        for (int d = 0; d < 6; ++d) o[d] = DIM == 3 ? u[d] : (d < 2 ? u[d] : (d == 5 ? u[2] : 0.0));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    __shared__ double vm[32];
    if ((lt & 31) == 0) vm[lt >> 5] = vmax;
    __syncthreads();
    if (lt == 0) {
        for (int w = 0; w < BT / 32; ++w) vmax = fmax(vmax, vm[w]);
        if (CS > 1) share<CS>(&Q.vmax[rank], vmax);
    }
    if (CS > 1) cluster_sync();  // also: no CTA leaves while another may still write into its shared memory
    if (rank == 0 && lt == 0) {
        for (int r = 0; r < CS; ++r)
            if (CS > 1) vmax = fmax(vmax, Q.vmax[r]);
        BatchSceneStats& st = B.stats[sc];
        st.contacts = nc;
        st.iterations = S.ite;
        st.fp32_iterations = 0;
        st.backtracks = S.nbt;
        st.restarts = S.nrs;
        st.corrections = 0;
        st.converged = S.conv && !S.err;
        st.violation = vmax;
    }
}

// Clusters of CS CTAs: cluster q < n_big solves the q-th largest scene with all of them, every
// later one CS of the other scenes, one per CTA (those never meet a cluster barrier).
template <int DIM, int CS>
__global__ void __launch_bounds__(kBatchFricThreads<DIM>, 1) k_fric_batch(FricArgs<double> A, BatchFricScenes B) {
    __shared__ ApgdState S;
    __shared__ SceneSums Q;
    if (A.sizes->overflow) return;  // the step is redone after the buffers grow (all CTAs alike)
    const int q = blockIdx.x / CS, rank = blockIdx.x % CS;
    if (q < B.n_big) {
        fric_scene<DIM, CS, kBatchFricThreads<DIM>>(A, B, B.order[q], rank, S, Q);
    } else {
        const int j = B.n_big + CS * (q - B.n_big) + rank;
        if (j < B.n_scenes) fric_scene<DIM, 1, kBatchFricThreads<DIM>>(A, B, B.order[j], 0, S, Q);
    }
}
// One CTA of BT threads per scene, PER of them on an SM: more scenes than the SMs hold at once.
template <int DIM, int BT, int PER>
__global__ void __launch_bounds__(BT, PER) k_fric_many(FricArgs<double> A, BatchFricScenes B) {
    __shared__ ApgdState S;
    __shared__ SceneSums Q;
    if (A.sizes->overflow) return;
    fric_scene<DIM, 1, BT>(A, B, B.order[blockIdx.x], 0, S, Q);
}

// ------------------------------------------------------------------ packing
template <typename T, int DIM>
__global__ void k_fric_pack(const Sizes* sizes, long long cap, const int* ci, const int* cj, const double* bP,
                            const double* bn, const double* cvec, int2* cij, Q4<T>* rec) {
    using F = FricShape<T, DIM>;
    GRID_STRIDE(c, sizes->C) {
        T r[F::row];
        const double* P = bP + 18 * c;
        if (DIM == 3) {
            for (int e = 0; e < 18; ++e) r[e] = (T)P[e];
        } else {
            r[0] = (T)P[6];
            r[1] = (T)P[7];
            r[2] = (T)P[15];
            r[3] = (T)P[16];
        }
        for (int d = 0; d < DIM; ++d) {
            r[F::at_n + d] = (T)bn[3 * c + d];
            r[F::at_c + d] = (T)cvec[3 * c + d];
        }
        cij[c] = make_int2(ci[c], cj[c]);
#pragma unroll
        for (int v = 0; v < F::nv; ++v) {
            Q4<T> q;
            T* o = reinterpret_cast<T*>(&q);
            for (int e = 0; e < F::per; ++e) o[e] = r[v * F::per + e];
            rec[v * cap + c] = q;
        }
    }
}
// another linear term in rows already packed (the FP32 correction solves; the FP64 correction and
// every fixed-point solve pack their rows anew)
template <typename T, int DIM>
__global__ void k_fric_pack_c(const Sizes* sizes, long long cap, const double* cvec, Q4<T>* rec) {
    using F = FricShape<T, DIM>;
    T* r = reinterpret_cast<T*>(rec);
    GRID_STRIDE(c, sizes->C) {
        for (int d = 0; d < DIM; ++d) {
            const int e = F::at_c + d;
            r[((e / F::per) * cap + c) * F::per + e % F::per] = (T)cvec[3 * c + d];
        }
    }
}
template <typename T, int DIM>
__device__ __forceinline__ void store_inc(unsigned e, const double* bP, Q4<T>* inc, long long at, int vs) {
    using F = FricShape<T, DIM>;
    const long long c = e & 0x7fffffffu;
    const int side = (int)(e >> 31);
    const double* P = bP + 18 * c + 9 * side;
    const T sg = side == 0 ? (T)1 : (T)-1;
    T r[F::inc];
    for (int q = 0; q < F::inc; ++q) r[q] = (T)0;
    if (DIM == 3) {
        for (int q = 0; q < 9; ++q) r[q] = sg * (T)P[q];
    } else {
        r[0] = sg * (T)P[6];
        r[1] = sg * (T)P[7];
    }
    r[F::at_idx] = fidx_bits<T>(e);
#pragma unroll
    for (int v = 0; v < F::ni; ++v) {
        Q4<T> q;
        T* o = reinterpret_cast<T*>(&q);
        for (int j = 0; j < F::per; ++j) o[j] = r[v * F::per + j];
        inc[at + v * vs] = q;
    }
}
template <typename T, int DIM>
__global__ void k_fric_pack_inc(int na, const int* ptr, const int* idx, const double* bP, Q4<T>* inc, long long slots,
                                const Sizes* sizes) {
    using F = FricShape<T, DIM>;
    const IncLayout lay = inc_layout(sizes, na, slots);
    if (lay.width) {
        const long long tot = (long long)lay.width * 32 * ((na + 31) / 32);
        GRID_STRIDE(t, tot) {
            const long long row = t >> 5, g = row / lay.width, p = g * 32 + (t & 31);
            const int r = (int)(row - g * lay.width);
            if (p >= na) continue;
            const int k0 = ptr[p];
            if (r < ptr[p + 1] - k0)
                store_inc<T, DIM>((unsigned)idx[k0 + r], bP, inc, row * F::ni * 32 + (t & 31), 32);
        }
        return;
    }
    const long long tot = ptr[na];
    GRID_STRIDE(k, tot) store_inc<T, DIM>((unsigned)idx[k], bP, inc, k * F::ni, 1);
}

int blocks(long long n) {
    const long long b = (n + 255) / 256;
    return (int)std::max<long long>(1, std::min<long long>(b, 16 * kSMs));
}

template <typename T, int DIM>
cudaError_t launch_fric_t(FricArgs<T>& A, int nblocks, cudaStream_t s) {
    cudaLaunchAttribute attr[1];
    if (nblocks <= kMaxCluster && !A.stall) {
        // small solves as one cluster (the wait-limit test needs the barrier that has a limit);
        // blocks past the last contact and body only take part in the barriers
        static ClusterAble able;
        const int lg = log2_up(nblocks);
        const cudaLaunchConfig_t cfg = cluster_config(1 << lg, FricThreads<T>::value, s, attr);
        if (cluster_fits(k_apgd_fric<T, DIM, true>, cfg, able, lg)) {
            if (cudaLaunchKernelEx(&cfg, k_apgd_fric<T, DIM, true>, A) == cudaSuccess) {
                g_fric_launches += 1;
                return cudaSuccess;
            }
            cudaGetLastError();  // refused (nothing ran): the cooperative form
        }
    }
    g_fric_launches += 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(FricThreads<T>::value);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_apgd_fric<T, DIM, false>, A);
}

}  // namespace

size_t fric_rec_bytes(int dim, bool fp32) { return (dim == 3 ? 24 : 8) * (fp32 ? 4 : 8); }
size_t fric_inc_bytes(int dim, bool fp32) { return dim == 3 ? (fp32 ? 48 : 80) : (fp32 ? 16 : 32); }
size_t fric_lam_bytes(int dim, bool fp32) { return (dim == 3 ? 4 : 2) * (fp32 ? 4 : 8); }
int fric_u_vectors(int dim) { return dim == 3 ? 2 : 1; }

int apgd_fric_max_blocks() {
    int dev = 0, sms = kSMs;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::min(sms, kSumMaxBlocks);  // one block per SM
}

template <typename T>
void launch_fric_pack(int dim, int na, const Contacts& c, const Assembly& a, const Incidence& inc, FricSolve<T>& f,
                      const Sizes* sizes, cudaStream_t s) {
    Q4<T>* rec = static_cast<Q4<T>*>(f.rec);
    Q4<T>* iv = static_cast<Q4<T>*>(f.inc);
    if (dim == 3) {
        k_fric_pack<T, 3><<<blocks(f.cap), 256, 0, s>>>(sizes, f.cap, c.ci, c.cj, a.bP, a.bn, a.cvec, f.cij, rec);
        k_fric_pack_inc<T, 3><<<blocks(f.inc_slots), 256, 0, s>>>(na, inc.ptr, inc.idx, a.bP, iv, f.inc_slots,
                                                                     sizes);
    } else {
        k_fric_pack<T, 2><<<blocks(f.cap), 256, 0, s>>>(sizes, f.cap, c.ci, c.cj, a.bP, a.bn, a.cvec, f.cij, rec);
        k_fric_pack_inc<T, 2><<<blocks(f.inc_slots), 256, 0, s>>>(na, inc.ptr, inc.idx, a.bP, iv, f.inc_slots,
                                                                     sizes);
    }
    g_fric_launches += 2;
}
template <typename T>
void launch_fric_pack_c(int dim, const double* cvec, FricSolve<T>& f, const Sizes* sizes, cudaStream_t s) {
    Q4<T>* rec = static_cast<Q4<T>*>(f.rec);
    if (dim == 3)
        k_fric_pack_c<T, 3><<<blocks(f.cap), 256, 0, s>>>(sizes, f.cap, cvec, rec);
    else
        k_fric_pack_c<T, 2><<<blocks(f.cap), 256, 0, s>>>(sizes, f.cap, cvec, rec);
    g_fric_launches += 1;
}
namespace {
template <typename T>
FricArgs<T> fric_args(int nin, int na, const ApgdSettings& st, const FricSolve<T>& f, const Sizes* sizes) {
    FricArgs<T> A;
    A.nin = nin;
    A.na = na;
    A.cap = f.cap;
    A.cij = f.cij;
    A.rec = static_cast<const Q4<T>*>(f.rec);
    A.shift = f.shift;
    A.inc_ptr = f.inc_ptr;
    A.inc = static_cast<const Q4<T>*>(f.inc);
    A.inc_slots = f.inc_slots;
    A.invm = reinterpret_cast<const V4<T>*>(f.invm);
    for (int k = 0; k < 3; ++k) A.lam[k] = f.lam[k];
    A.u0 = f.u[0];
    A.u1 = f.u[1];
    A.u2 = f.u[2];
    A.u3 = f.u[3];
    A.qv = f.qv;
    A.wu = f.wu;
    A.lam_out = f.lam_out;
    A.u_out = f.u_out;
    A.sums = f.sums;
    A.bar = f.barrier;
    A.result = f.result;
    A.sizes = sizes;
    A.alpha = st.alpha;
    A.tol = st.tol;
    A.dt2 = st.dt * st.dt;
    A.mu = st.mu;
    A.max_ite = st.max_ite;
    A.dynamic = st.dynamic;
    A.curvature_start = st.curvature_start;
    A.stall = st.stall;
    return A;
}
}  // namespace

template <typename T>
cudaError_t launch_apgd_fric(int nin, int na, int dim, const ApgdSettings& st, FricSolve<T>& f, const Sizes* sizes,
                             int nblocks, cudaStream_t s) {
    FricArgs<T> A = fric_args<T>(nin, na, st, f, sizes);
    return dim == 3 ? launch_fric_t<T, 3>(A, nblocks, s) : launch_fric_t<T, 2>(A, nblocks, s);
}

// ------------------------------------------------------------------ how a batch is split
// One iteration of a scene of n bodies costs max(floor, base + slope n) microseconds (its contacts
// follow its bodies: 2.5 a disk, 3.8 a sphere).  Measured, clusters on one scene, the others with
// every SM at work:
//                                     2D, n = 30   100   300  1000  2500    3D, n = 30   100   300  1000
//   cluster of 4                            5.5   5.8   7.8  11.2  20.7            7.2   9.2  15.2  24.5
//   cluster of 2                            5.4   5.9   8.2  13.2  29.1            7.3   9.9  17.9  40.0
//   one CTA an SM                           4.1   4.5   7.6  18.0  42.3            5.0   9.0  21.0  62.3
//   2D two CTAs of 256 an SM                4.0   4.8  10.8
//   2D four, 3D two CTAs of 128 an SM       4.3   6.7  19.5                        6.0  12.7
// Clusters shorten the longest scene; more and smaller CTAs get more scenes through.  The form whose
// list schedule of the scenes, largest first, ends first is taken.  Milliseconds a step of the generic
// 6-dof rows (two CTAs of 256 an SM), of clusters of two whatever the number of scenes, and of this
// rule: 1000 x 30 disks 12.1, 39.4, 5.3; 600 x 100 18.1, 29.2, 7.2; 300 x 400 34.6, 23.5, 14.5;
// 1000 x 30 spheres 16.7, 55.9, 12.7; 300 x 200 29.6, 40.2, 24.4.
namespace {
struct IterationCost {
    double floor, base, slope;
    double of(int n) const { return std::max(floor, base + slope * n); }
};
struct FricForm {
    int cs, per_sm;  // CTAs of a cluster; CTAs of an SM
    IterationCost large, other;  // a scene on a cluster, on one CTA
};
const FricForm kFricForms[2][FricBatchForm::kCount] = {
    {{4, 1, {5.5, 5.0, 0.0063}, {4.1, 2.6, 0.0165}},
     {2, 1, {5.4, 4.8, 0.0098}, {4.1, 2.6, 0.0165}},
     {2, 1, {}, {4.1, 2.6, 0.0165}},
     {1, 2, {}, {4.0, 1.8, 0.0300}},
     {1, 4, {}, {4.3, 0.3, 0.0640}}},
    {{4, 1, {7.2, 8.5, 0.0160}, {5.0, 1.0, 0.0750}},
     {2, 1, {7.3, 7.0, 0.0350}, {5.0, 1.0, 0.0750}},
     {2, 1, {}, {5.0, 1.0, 0.0750}},
     {0, 0, {}, {}},  // 256 threads with a 3D row each fill the registers of an SM
     {1, 2, {}, {5.9, 0.0, 0.1320}}}};

template <int DIM, int CS>
cudaLaunchConfig_t fric_cluster_config(int clusters, cudaStream_t s, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = cluster_config(CS, kBatchFricThreads<DIM>, s, at);
    cfg.gridDim = dim3(CS * clusters);
    return cfg;
}
// clusters of CS CTAs that run at once (an SM group need not be a multiple of four: 37 clusters of
// four on 148 SMs take two rounds)
template <int DIM, int CS>
int fric_cluster_slots() {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = fric_cluster_config<DIM, CS>(kSMs / CS, nullptr, at);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_fric_batch<DIM, CS>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return kSMs / CS;
    }
    return n;
}

// when the last of the CTAs (clusters) that start in order on `slots` free places ends
double list_schedule(const std::vector<double>& cost, int slots) {
    std::priority_queue<double, std::vector<double>, std::greater<double>> busy;
    double end = 0.0;
    for (double c : cost) {
        double at = 0.0;
        if ((int)busy.size() == slots) {
            at = busy.top();
            busy.pop();
        }
        busy.push(at + c);
        end = std::max(end, at + c);
    }
    return end;
}
}  // namespace

FricBatchForm fric_batch_form(int dim, const std::vector<int>& bodies) {
    FricBatchForm best{};
    double least = 0.0;
    int big = 0;  // the scenes with at least half the largest one's bodies
    while (big < (int)bodies.size() && 2LL * bodies[big] >= bodies[0]) ++big;
    const int slots4 = dim == 3 ? fric_cluster_slots<3, 4>() : fric_cluster_slots<2, 4>();
    const int slots2 = dim == 3 ? fric_cluster_slots<3, 2>() : fric_cluster_slots<2, 2>();
    for (int k = 0; k < FricBatchForm::kCount; ++k) {
        const FricForm& f = kFricForms[dim == 3][k];
        if (f.cs == 0) continue;
        const int n_big = k == FricBatchForm::kCluster4 || k == FricBatchForm::kCluster2 ? big : 0;
        std::vector<double> cost;
        for (int j = 0; j < (int)bodies.size(); j += j < n_big ? 1 : f.cs) {
            // the iterations of like scenes differ by about a fifth either way
            const double x = j * 0.6180339887498949, spread = 0.8 + 0.4 * (x - std::floor(x));
            cost.push_back(spread * (j < n_big ? f.large.of(bodies[j]) : f.other.of(bodies[j])));
        }
        const double t = list_schedule(cost, f.cs == 4 ? slots4 : f.cs == 2 ? slots2 : kSMs * f.per_sm);
        if (k == 0 || t < least) {
            least = t;
            best.form = k;
            best.n_big = n_big;
        }
    }
    return best;
}

namespace {
template <int DIM, int CS>
cudaError_t launch_fric_clusters(const FricArgs<double>& A, const BatchFricScenes& B, cudaStream_t s) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg =
        fric_cluster_config<DIM, CS>(B.n_big + (B.n_scenes - B.n_big + CS - 1) / CS, s, at);
    return cudaLaunchKernelEx(&cfg, k_fric_batch<DIM, CS>, A, B);
}
template <int DIM, int BT, int PER>
cudaError_t launch_fric_many(const FricArgs<double>& A, const BatchFricScenes& B, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B.n_scenes);
    cfg.blockDim = dim3(BT);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, k_fric_many<DIM, BT, PER>, A, B);
}
}  // namespace

cudaError_t launch_fric_batch(int nin, int na, int dim, const ApgdSettings& st, FricSolve<double>& f,
                              const Sizes* sizes, BatchFricScenes B, FricBatchForm form, cudaStream_t s) {
    if (B.n_scenes <= 0) return cudaSuccess;
    const FricArgs<double> A = fric_args<double>(nin, na, st, f, sizes);
    B.n_big = std::min(std::max(form.n_big, 0), B.n_scenes);
    g_fric_launches += 1;
    switch (form.form) {
        case FricBatchForm::kCluster4:
            return dim == 3 ? launch_fric_clusters<3, 4>(A, B, s) : launch_fric_clusters<2, 4>(A, B, s);
        case FricBatchForm::kMany256:
            return launch_fric_many<2, 256, 2>(A, B, s);
        case FricBatchForm::kMany128:
            return dim == 3 ? launch_fric_many<3, 128, 2>(A, B, s) : launch_fric_many<2, 128, 4>(A, B, s);
        default:
            return dim == 3 ? launch_fric_clusters<3, 2>(A, B, s) : launch_fric_clusters<2, 2>(A, B, s);
    }
}
#define INST(T) \
    template void launch_fric_pack<T>(int, int, const Contacts&, const Assembly&, const Incidence&, FricSolve<T>&, \
                                      const Sizes*, cudaStream_t); \
    template void launch_fric_pack_c<T>(int, const double*, FricSolve<T>&, const Sizes*, cudaStream_t); \
    template cudaError_t launch_apgd_fric<T>(int, int, int, const ApgdSettings&, FricSolve<T>&, const Sizes*, int, \
                                             cudaStream_t);
INST(float) INST(double)
#undef INST

}  // namespace scopi_gpu
