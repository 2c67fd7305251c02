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
#include <algorithm>

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

__device__ __forceinline__ void put4(float* o, const float4& v) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void put4(double* o, const double2& v) { o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void fld4(const float4* p, float* o) { put4(o, *p); }
__device__ __forceinline__ void fld4(const dvec4* p, double* o) {
    const double2* q = reinterpret_cast<const double2*>(p);
    put4(o, q[0]);
    put4(o + 2, q[1]);
}
__device__ __forceinline__ void fld4cg(const float4* p, float* o) { put4(o, __ldcg(p)); }
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
// roundings written out where the compiler could contract in more than one way: a solve's
// bits are then the same whatever kernel it runs in
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
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
    V4<T>* lam0;
    V4<T>* lam1;
    V4<T>* lam2;
    V4<T>* u0;
    V4<T>* u1;
    V4<T>* u2;
    V4<T>* u3;
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

template <typename T>
__device__ __forceinline__ V4<T>* pick_lam(const FricArgs<T>& A, int k) {
    return k == 0 ? A.lam0 : (k == 1 ? A.lam1 : A.lam2);
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
// u of a body, written by other blocks: (v, w), 2D (vx, vy, w)
template <typename T, int DIM>
__device__ __forceinline__ void gather_u(const V4<T>* u, int p, T* o) {
    T t[4];
    fld4cg(u + (long long)p * FricShape<T, DIM>::nu, t);
    o[0] = t[0];
    o[1] = t[1];
    o[2] = t[2];
    if (DIM == 3) {
        fld4cg(u + 2ll * p + 1, t);
        o[3] = t[0];
        o[4] = t[1];
        o[5] = t[2];
    }
}
// this thread's own body
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
template <typename T, int DIM>
__device__ __forceinline__ void contact_row(const T* r, const T* ui, const T* uj, const T* lam, const T* lprev,
                                            T beta, bool use_prev, bool bt, double alpha, double mu, T dt2,
                                            const double* shift, T* lout, double* s) {
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
}

// w = A^T l+ of one body over its n incidences, KB records and multipliers in flight
template <typename T, int DIM, int KB>
__device__ __forceinline__ void body_force(const Q4<T>* inc, const IncWalk& wk, const V4<T>* lnew, int n, T* w) {
    using F = FricShape<T, DIM>;
#pragma unroll
    for (int d = 0; d < F::dof; ++d) w[d] = (T)0;
    for (int kb = 0; kb < n; kb += KB) {
        T e[KB][F::inc], l[KB][4];
#pragma unroll
        for (int q = 0; q < KB; ++q)
            if (kb + q < n)
#pragma unroll
                for (int v = 0; v < F::ni; ++v)
                    put4(e[q] + v * F::per, inc[wk.first + (long long)(kb + q) * wk.rs + v * wk.vs]);
#pragma unroll
        for (int q = 0; q < KB; ++q)
            if (kb + q < n) fld4cg(lnew + (fidx(e[q][F::at_idx]) & 0x7fffffffu), l[q]);
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

// Threads per block (one block per SM).  FP64 keeps the 256 threads whose per-thread sums its
// decisions have always been taken from; FP32 decisions do not hang on the last bits.
constexpr long long kMaxBacktracks = 4000;

template <typename T>
struct FricThreads {
    static constexpr int value = sizeof(T) == 4 ? 512 : 256;
    static constexpr int kb = sizeof(T) == 4 ? 3 : 3;
};

template <typename T, int DIM>
__global__ void __launch_bounds__(FricThreads<T>::value, 1) k_apgd_fric(FricArgs<T> A) {
    using F = FricShape<T, DIM>;
    constexpr int KB = FricThreads<T>::kb;
    __shared__ ApgdState S;
    __shared__ double red[8][32];
    const int tid = threadIdx.x;
    const int C = A.sizes->C;
    const IncLayout lay = inc_layout(A.sizes, A.na, A.inc_slots);
    GridSums<false> G{A.sums, gridDim.x, A.bar, 0u, A.stall != 0 && blockIdx.x == 0};
    if (tid == 0) state_init(S, A.alpha);
    __syncthreads();
    if (A.curvature_start) {
        // initial step from the curvature along the first projected-gradient direction d of the
        // cold start (in the candidate buffer, which the first contact pass overwrites), with
        // 256 threads per block: the sums set the step, so their order is kept in FP32 too
        const long long S0 = (long long)gridDim.x * 256, b0 = (long long)blockIdx.x * 256 + tid;
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
                fst4(A.lam2 + c, v);
            }
        double t1 = 0.0, t6 = 0.0;
        block_sum<2>(a);
        bool ok = G.exchange(a[0], t1);
        double b[2] = {0.0, 0.0};
        if (ok && tid < 256)
            for (long long p = b0; p < A.na; p += S0) {
                T w[F::dof], u[F::dof], im[4];
                const int k0 = A.inc_ptr[p];
                body_force<T, DIM, KB>(A.inc, inc_walk(lay, F::ni, p, k0), A.lam2, A.inc_ptr[p + 1] - k0, w);
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
    for (;;) {
        if (S.done) break;
        const double alpha = S.alpha;
        const bool bt = S.bt != 0, use_prev = S.use_prev != 0;
        const T beta = (T)S.beta;
        const V4<T>* lam = pick_lam(A, S.il);
        const V4<T>* lprev = pick_lam(A, S.ip);
        V4<T>* lnew = pick_lam(A, S.in_);
        const V4<T>* uY = pick_u(A, S.jY);
        {
            double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            int2 ij = base < C ? A.cij[base] : make_int2(0, 0);
#pragma unroll 1
            for (long long c = base; c < C; c += S_) {
                const int2 me = ij;
                if (c + S_ < C) ij = A.cij[c + S_];
                T ui[F::dof], uj[F::dof], r[F::row], lm[4], lq[4], lo[3];
#pragma unroll
                for (int d = 0; d < F::dof; ++d) ui[d] = uj[d] = (T)0;
                if (me.x >= A.nin) gather_u<T, DIM>(uY, me.x - A.nin, ui);
                if (me.y >= A.nin) gather_u<T, DIM>(uY, me.y - A.nin, uj);
                load_row<T, DIM>(A.rec, A.cap, c, r);
                fld4(lam + c, lm);
                if (use_prev) fld4(lprev + c, lq);
                contact_row<T, DIM>(r, ui, uj, lm, lq, beta, use_prev, bt, alpha, A.mu, (T)A.dt2,
                                    A.shift ? A.shift + 3 * c : nullptr, lo, s);
                fst4(lnew + c, lo);
            }
            constexpr int NS = sizeof(T) == 4 ? 4 : 8;
            G.template publish<NS>(s, red);
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
            const V4<T>* uL = pick_u(A, S.jL);
            V4<T>* uN = pick_u(A, S.jN);
            V4<T>* uYN = pick_u(A, S.jYN);
            const T bn_ = (T)S.beta_n;
            double s[1] = {0.0};
#pragma unroll 1
            for (long long p = base; p < A.na; p += S_) {
                const int k0 = A.inc_ptr[p], k1 = A.inc_ptr[p + 1];
                T im[4], ul[F::dof], uy[F::dof], w[F::dof], u[F::dof];
                fld4(A.invm + p, im);
                if (bn_ != (T)0) load_u<T, DIM>(uL, p, ul);
                if (sizeof(T) == 4) load_u<T, DIM>(uY, p, uy);
                body_force<T, DIM, KB>(A.inc, inc_walk(lay, F::ni, p, k0), lnew, k1 - k0, w);
                body_velocity<T, DIM>(im, w, u);
                store_u<T, DIM>(uN, p, u);
                // w.u gives F(l+) for the reference's test (FP64); FP32 tests the curvature
                if (sizeof(T) == 8)
                    s[0] += body_wu<T, DIM>(w, u);
                else
                    s[0] += body_curvature<T, DIM>(im, u, uy);
                if (bn_ != (T)0) {
#pragma unroll
                    for (int d = 0; d < F::dof; ++d) u[d] = fma_rn(bn_, add_rn(u[d], -ul[d]), u[d]);
                }
                store_u<T, DIM>(uYN, p, u);
            }
            G.template publish<1>(s, red);
            if (tid < 32) {
                const NextStep ns = prepare_step<T>(S, A.tol);
                double t[1];
                const bool ok = G.template collect<1>(t);
                if (tid == 0) {
                    if (!ok) {
                        S.err = 1;
                        S.done = 1;
                    } else {
                        decide_step<T>(S, t[0], t[0], A.dt2, A.dynamic, A.max_ite, ns, kMaxBacktracks);
                    }
                }
            }
            G.next();
            __syncthreads();
        }
    }
    // the result, in the layouts of the other kernels (every thread its own contacts and bodies)
    const V4<T>* lres = pick_lam(A, S.il);
    const V4<T>* ures = pick_u(A, S.jL);
    for (long long c = base; c < C; c += S_) {
        T l[4];
        fld4(lres + c, l);
        for (int d = 0; d < 3; ++d) A.lam_out[3 * c + d] = l[d];
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
// another linear term in rows already packed (correction and fixed-point solves)
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
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(FricThreads<T>::value);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    g_fric_launches += 1;
    return cudaLaunchKernelEx(&cfg, k_apgd_fric<T, DIM>, A);
}

}  // namespace

size_t fric_rec_bytes(int dim, bool fp32) { return (dim == 3 ? 24 : 8) * (fp32 ? 4 : 8); }
size_t fric_inc_bytes(int dim, bool fp32) { return dim == 3 ? (fp32 ? 48 : 80) : (fp32 ? 16 : 32); }
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
template <typename T>
cudaError_t launch_apgd_fric(int nin, int na, int dim, const ApgdSettings& st, FricSolve<T>& f, const Sizes* sizes,
                             int nblocks, cudaStream_t s) {
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
    A.lam0 = f.lam[0];
    A.lam1 = f.lam[1];
    A.lam2 = f.lam[2];
    A.u0 = f.u[0];
    A.u1 = f.u[1];
    A.u2 = f.u[2];
    A.u3 = f.u[3];
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
    return dim == 3 ? launch_fric_t<T, 3>(A, nblocks, s) : launch_fric_t<T, 2>(A, nblocks, s);
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
