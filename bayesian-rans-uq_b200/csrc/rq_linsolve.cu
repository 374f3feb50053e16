// Standalone batched linear solves on the device: one thread-block cluster per LDU system
// (1 to 16 CTAs by its rows and the batch), persistent clusters pulling systems from a queue
// (largest first, as the host orders them). The solvers restate core/include/LinearSolver.hpp:
//   PCG (:184-246) with the Jacobi preconditioner or the AMG V-cycle of this
//   project (damped-Jacobi smoothing, aggregate-sum restriction, aggregate
//   broadcast prolongation scaled by an over-correction factor, dense coarsest
//   inverse), right-Jacobi BiCGSTAB
//   (:251-345), and a mixed form: FP32 PCG corrections inside an FP64
//   residual-refinement loop.
// Level 0 keeps the reference's matvec order per row (diagonal, then faces in
// increasing index); coarse levels are column-sorted. Every dot product
// and norm is an FP64 block reduction whose result all threads share, so
// control flow is uniform.
//
// What bounds it: a large system streams its rows and vectors from HBM or L2, a small one
// is a chain of phases of a microsecond each. Rows are stored in slices of 32, so that a
// warp's loads of entry k are consecutive; a damped-Jacobi sweep is one pass from one
// vector to another; the levels of up to 2048 rows run whole in every CTA of the cluster,
// on vectors in its shared memory and with its own barrier (about 80 cycles against 500).
#include "rq_lin.cuh"

#include <cuda_runtime.h>

namespace rq {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr double kOmega = 0.75; // damped-Jacobi weight of the V-cycle smoother
// Scale of the coarse-grid correction: piecewise-constant prolongation under-
// corrects smooth error, and over-correcting by 1.7 cuts the PCG iterations of
// the log-normal Poisson systems from 100 to 30 at 256 x 256 (CPU restatement).
constexpr double kAlpha = 1.7;
constexpr int kSweeps = 2;     // pre- and post-smoothing sweeps
constexpr int kMixedRounds = 12;
constexpr double kMixedInnerTol = 1e-4; // relative drop asked of each FP32 correction

// NT: threads of a CTA; the smaller ones solve systems of one slice
template <int NT> struct LinShared {
    static constexpr bool kOne = NT == kLinSmallThreads;
    __device__ int nCtas() const { return kOne ? 1 : ctas; }
    __device__ int nSlices() const { return kOne ? 1 : sys.slices; }
    DevLinSys sys;
    double red[kOne ? 4 : 2 * kLinMaxSlices][NT / 32]; // warp sums of the CTA's slices
    double cred[2][2][kOne ? 1 : kLinMaxSlices]; // the slices' sums, in alternating buffers
    int job;
    int rank, ctas;
};
extern __shared__ __align__(16) unsigned char linSmem[]; // vectors of the local levels

// thread index in the cluster and its threads; the cluster's barrier
template <int NT> __device__ __forceinline__ int gTid(const LinShared<NT> &S) {
    return (S.kOne ? 0 : S.rank * NT) + threadIdx.x;
}
template <int NT> __device__ __forceinline__ int gThreads(const LinShared<NT> &S) { return S.nCtas() * NT; }
template <int NT> __device__ __forceinline__ void gSync(const LinShared<NT> &S) {
    if (S.nCtas() > 1)
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    else
        __syncthreads();
}
template <typename V> __device__ __forceinline__ void putRemote(V *p, V v, int rank) {
    unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p)), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    if constexpr (sizeof(V) == 8)
        asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(r), "l"(__double_as_longlong(v)) : "memory");
    else
        asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(r), "r"(static_cast<int>(v)) : "memory");
}

// Sums over the rows of a system. They are formed in sys.slices slices, whatever the number of
// CTAs: slice i holds the rows (i + k slices) NT + 0 .. NT - 1, k = 0, 1, ..., and CTA r of c
// the slices r, r + c, ..., which are the rows of its other passes too. A thread adds its rows
// of a slice, each warp its threads by shuffles (lane 0 parks the sum), one warp per slice and
// value the warps, and every thread the slices in order: all threads return the same bits, and
// so does a cluster of any size. (With one slice every warp adds the warps, which saves a
// barrier; the parked sums alternate between two buffers then.)
__device__ __forceinline__ double addLanes(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    return v;
}
// rows(t0, nt) adds the terms of the rows t0, t0 + nt, ... to v
template <int K, int NT, typename Rows>
__device__ __forceinline__ void parkOver(double (&v)[K], LinShared<NT> &S, int rp, Rows rows) {
    const int nt = S.nSlices() * NT, own = S.nSlices() / S.nCtas();
    const int first = S.nSlices() == 1 ? rp * K : 0;
    for (int i = 0; i < own; ++i) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            v[k] = 0.0;
        rows(i * S.nCtas() * NT + gTid(S), nt);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double w = addLanes(v[k]);
            if ((threadIdx.x & 31) == 0)
                S.red[first + i * K + k][threadIdx.x >> 5] = w;
        }
    }
}
// the sums of what parkOver left; a barrier of the cluster for what was stored before
template <int K, int NT>
__device__ __forceinline__ void totalSums(double (&v)[K], LinShared<NT> &S, int &rp) {
    const int lane = threadIdx.x & 31;
    __syncthreads();
    if (S.nSlices() == 1) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            v[k] = addLanes(lane < NT / 32 ? S.red[rp * K + k][lane] : 0.0);
        rp ^= 1;
        return;
    }
    const int rows = S.sys.slices / S.ctas * K;
    for (int t = threadIdx.x >> 5; t < rows; t += NT / 32) {
        const double w = addLanes(lane < NT / 32 ? S.red[t][lane] : 0.0);
        const int i = t / K, k = t - i * K;
        if (lane < S.ctas)
            putRemote(&S.cred[rp][k][i * S.ctas + S.rank], w, lane);
    }
    gSync(S);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        v[k] = S.cred[rp][k][0];
        for (int c = 1; c < S.sys.slices; ++c)
            v[k] += S.cred[rp][k][c];
    }
    rp ^= 1;
}
template <int K, int NT, typename Rows>
__device__ __forceinline__ void sumOver(double (&v)[K], LinShared<NT> &S, int &rp, Rows rows) {
    parkOver(v, S, rp, rows);
    totalSums(v, S, rp);
}
static_assert(kLinThreads <= 1024, "a lane per warp sum");

// one level of the hierarchy in value type T (FP64, or the FP32 copies)
template <typename T> struct Lv {
    int n, nc, sh;
    const int *ptr, *col;
    const T *val, *rdg;
    const int *agg, *childPtr, *childIdx;
    T *b, *x, *r; // workspace vectors (levels >= 1; level 0 uses the caller's)
};

// use(i, row i times x) for the rows t0, t0 + nt, ...; entries in order. The first five columns
// and values (a grid system's row) are loaded before the first is used. (Two rows at a time
// with 1024 threads, two or four with 512: 2 to 18 % slower at every size but 512 x 512 with
// 1024 threads, 1 % slower there; the registers spill or the warps are too few.)
template <typename T, typename Use>
__device__ __forceinline__ void passRows(const Lv<T> &A, const T *x, int t0, int nt, Use use) {
    constexpr int B = 5;
    const int step = 1 << A.sh;
    for (int i = t0; i < A.n; i += nt) {
        const int k1 = __ldg(A.ptr + (i >> A.sh) + 1);
        T s = T(0);
        for (int e = __ldg(A.ptr + (i >> A.sh)) + (i & (step - 1)); e < k1; e += B * step) {
            int c[B];
            T v[B], xc[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const bool in = e + u * step < k1;
                c[u] = in ? __ldg(A.col + e + u * step) : -1;
                v[u] = in ? __ldg(A.val + e + u * step) : T(0);
            }
#pragma unroll
            for (int u = 0; u < B; ++u)
                xc[u] = c[u] >= 0 ? x[c[u]] : T(0);
#pragma unroll
            for (int u = 0; u < B; ++u)
                if (c[u] >= 0)
                    s += v[u] * xc[u];
        }
        use(i, s);
    }
}

template <typename T>
__device__ __forceinline__ Lv<T> levelOf(const DevLinSys &S, int l, void *ws) {
    const DevLinLevel &d = S.lev[l];
    T *w = static_cast<T *>(l >= S.loc ? static_cast<void *>(linSmem) : ws) + d.vecOff;
    Lv<T> A{d.n, d.nc, d.sh, d.ptr, d.col, nullptr, nullptr, d.agg, d.childPtr, d.childIdx,
            w, w + d.n, w + 2L * d.n};
    if constexpr (sizeof(T) == 8) {
        A.val = d.val;
        A.rdg = d.rdg;
    } else {
        A.val = d.val32;
        A.rdg = d.rdg32;
    }
    return A;
}

// z = M^-1 r by one V-cycle: damped Jacobi from zero, residual restricted by
// aggregate sums, the coarsest level by its dense inverse, the correction
// broadcast back and the same sweeps after it (a symmetric preconditioner).
// lvws: the level vectors of levels 1 .. loc - 1; t: a level-0 scratch vector. A level's
// iterate alternates between x and r; its solution ends in r (the coarsest's in x).
// Parks (r, z) (parkOver).
template <typename T, int NT>
__device__ void vcycle(LinShared<NT> &S, int rp, const T *r, T *z, T *t, void *lvws, const T *inv) {
    static_assert(kSweeps == 2, "the buffers alternate for two sweeps");
    const DevLinSys &sys = S.sys;
    const int L = sys.nlev;
    const T w = T(kOmega);
    double rz[1];
    if (L == 1) { // the whole system is the coarsest level
        const int m = sys.m;
        parkOver(rz, S, rp, [&](int t0, int nt) {
            for (int i = t0; i < m; i += nt) {
                T s = T(0);
                for (int j = 0; j < m; ++j)
                    s += inv[i * m + j] * r[j];
                z[i] = s;
                rz[0] += double(r[i]) * double(s);
            }
        });
        return;
    }
    auto tid = [&](int l) { return l >= sys.loc ? static_cast<int>(threadIdx.x) : gTid(S); };
    auto threads = [&](int l) { return l >= sys.loc ? NT : gThreads(S); };
    auto sync = [&](int l) {
        if (l >= sys.loc)
            __syncthreads();
        else
            gSync(S);
    };
    const T *fr = nullptr; // residual of the level above
    for (int l = 0; l + 1 < L; ++l) {
        Lv<T> A = levelOf<T>(sys, l, lvws);
        const int t0 = tid(l), nt = threads(l);
        const T *b = l == 0 ? r : A.b;
        T *x = l == 0 ? t : A.x, *y = l == 0 ? z : A.r;
        if (l == 0) {
            for (int i = t0; i < A.n; i += nt)
                x[i] = w * b[i] * __ldg(A.rdg + i);
        } else { // restricted right-hand side
            const Lv<T> F = levelOf<T>(sys, l - 1, lvws);
            for (int i = t0; i < A.n; i += nt) {
                T s = T(0);
                for (int k = __ldg(F.childPtr + i); k < __ldg(F.childPtr + i + 1); ++k)
                    s += fr[__ldg(F.childIdx + k)];
                A.b[i] = s;
                x[i] = w * s * __ldg(A.rdg + i);
            }
        }
        sync(l);
        passRows<T>(A, x, t0, nt, [&](int i, T ax) {
            const T res = b[i] - ax;
            y[i] = x[i] + w * res * __ldg(A.rdg + i);
        });
        sync(l);
        passRows<T>(A, y, t0, nt, [&](int i, T ax) { x[i] = b[i] - ax; });
        sync(l);
        fr = x;
    }
    const T *xc;
    {
        const int l = L - 1, t0 = tid(l), nt = threads(l);
        Lv<T> A = levelOf<T>(sys, l, lvws);
        const Lv<T> F = levelOf<T>(sys, l - 1, lvws);
        const int m = A.n;
        for (int i = t0; i < m; i += nt) {
            T s = T(0);
            for (int k = __ldg(F.childPtr + i); k < __ldg(F.childPtr + i + 1); ++k)
                s += fr[__ldg(F.childIdx + k)];
            A.b[i] = s;
        }
        sync(l);
        for (int i = t0; i < m; i += nt) {
            T s = T(0);
            for (int j = 0; j < m; ++j)
                s += inv[i * m + j] * A.b[j];
            A.x[i] = s;
        }
        sync(l);
        xc = A.x;
    }
    for (int l = L - 2; l >= 0; --l) {
        Lv<T> A = levelOf<T>(sys, l, lvws);
        const int t0 = tid(l), nt = threads(l);
        const T *b = l == 0 ? r : A.b;
        T *x = l == 0 ? t : A.x, *y = l == 0 ? z : A.r;
        for (int i = t0; i < A.n; i += nt)
            y[i] += T(kAlpha) * xc[__ldg(A.agg + i)];
        sync(l);
        passRows<T>(A, y, t0, nt, [&](int i, T ax) {
            const T res = b[i] - ax;
            x[i] = y[i] + w * res * __ldg(A.rdg + i);
        });
        sync(l);
        auto last = [&](int i, T ax) {
            const T res = b[i] - ax;
            const T zi = x[i] + w * res * __ldg(A.rdg + i);
            y[i] = zi;
            return zi;
        };
        if (l > 0) {
            passRows<T>(A, x, t0, nt, last);
            sync(l);
        } else { // the caller's sum ends with a barrier
            parkOver(rz, S, rp, [&](int s0, int st) {
                passRows<T>(A, x, s0, st, [&](int i, T ax) {
                    rz[0] += double(r[i]) * double(last(i, ax));
                });
            });
        }
        xc = y;
    }
}

// z = M^-1 r; returns (r, z)
template <typename T, int NT>
__device__ __forceinline__ double precondition(LinShared<NT> &S, int &rp, bool amg, const T *r, T *z,
                                               T *t, void *lvws, const T *inv, const T *rdg0) {
    double a[1];
    if (amg)
        vcycle<T>(S, rp, r, z, t, lvws, inv);
    else
        parkOver(a, S, rp, [&](int t0, int nt) {
            for (int i = t0; i < S.sys.n; i += nt) {
                const T zi = r[i] * __ldg(rdg0 + i);
                z[i] = zi;
                a[0] += double(r[i]) * double(zi);
            }
        });
    totalSums(a, S, rp);
    return a[0];
}

struct PcgOut {
    int iterations;
    bool converged;
    double finalRes;
};

// PCG from x (in T) with r = b - A x already in r and r0n = ||r||; the
// reference's loop (LinearSolver.hpp:206-245). Vectors r, z, p, q, t: n each.
template <typename T, int NT>
__device__ PcgOut pcg(LinShared<NT> &S, int &rp, const Lv<T> &A0, T *x, T *r, T *z, T *p, T *q, T *t,
                      void *lvws, const T *inv, double r0n, int maxIter, double tol, bool amg) {
    const int n = A0.n;
    PcgOut o{0, false, 0.0};
    double rz = precondition<T>(S, rp, amg, r, z, t, lvws, inv, A0.rdg);
    for (int i = gTid(S); i < n; i += gThreads(S))
        p[i] = z[i];
    gSync(S);
    for (int it = 0; it < maxIter; ++it) {
        double b1[1];
        sumOver(b1, S, rp, [&](int t0, int nt) {
            passRows<T>(A0, p, t0, nt, [&](int i, T v) {
                q[i] = v;
                b1[0] += double(p[i]) * double(v);
            });
        });
        const double pAp = b1[0];
        if (fabs(pAp) < 1e-30)
            break;
        const double alpha = rz / pAp;
        double b2[1];
        sumOver(b2, S, rp, [&](int t0, int nt) {
            for (int i = t0; i < n; i += nt) {
                x[i] += T(alpha) * p[i];
                const T ri = r[i] - T(alpha) * q[i];
                r[i] = ri;
                b2[0] += double(ri) * double(ri);
            }
        });
        o.iterations = it + 1;
        o.finalRes = sqrt(b2[0]) / r0n;
        if (o.finalRes < tol) {
            o.converged = true;
            return o;
        }
        const double rzNew = precondition<T>(S, rp, amg, r, z, t, lvws, inv, A0.rdg);
        const double beta = rzNew / (rz + 1e-30);
        for (int i = gTid(S); i < n; i += gThreads(S))
            p[i] = z[i] + T(beta) * p[i];
        gSync(S);
        rz = rzNew;
    }
    return o;
}

// Right-Jacobi BiCGSTAB (LinearSolver.hpp:251-345) in FP64; r holds b - A x.
template <int NT>
__device__ PcgOut bicgstab(LinShared<NT> &S, int &rp, const Lv<double> &A0, double *x, double *ws,
                           double r0n, int maxIter, double tol) {
    const int n = A0.n;
    double *r = ws, *rh = ws + n, *p = ws + 2L * n, *v = ws + 3L * n, *s = ws + 4L * n,
           *t = ws + 5L * n, *ph = ws + 6L * n, *sh = ws + 7L * n;
    PcgOut o{0, false, 0.0};
    double a[1];
    sumOver(a, S, rp, [&](int t0, int nt) {
        for (int i = t0; i < n; i += nt) {
            rh[i] = r[i];
            p[i] = 0.0;
            v[i] = 0.0;
            a[0] += r[i] * r[i];
        }
    });
    double rhoN = a[0], rho = 1, alpha = 1, omega = 1;
    for (int it = 0; it < maxIter; ++it) {
        if (fabs(rhoN) < 1e-30)
            break;
        const double beta = (rhoN / (rho + 1e-30)) * (alpha / (omega + 1e-30));
        for (int i = gTid(S); i < n; i += gThreads(S)) {
            const double pi = r[i] + beta * (p[i] - omega * v[i]);
            p[i] = pi;
            ph[i] = pi * __ldg(A0.rdg + i);
        }
        gSync(S);
        double a1[1];
        sumOver(a1, S, rp, [&](int t0, int nt) {
            passRows<double>(A0, ph, t0, nt, [&](int i, double vi) {
                v[i] = vi;
                a1[0] += rh[i] * vi;
            });
        });
        if (fabs(a1[0]) < 1e-30)
            break;
        alpha = rhoN / a1[0];
        double a2[1];
        sumOver(a2, S, rp, [&](int t0, int nt) {
            for (int i = t0; i < n; i += nt) {
                const double si = r[i] - alpha * v[i];
                s[i] = si;
                sh[i] = si * __ldg(A0.rdg + i);
                a2[0] += si * si;
            }
        });
        const double sn = sqrt(a2[0]);
        if (sn / r0n < tol) {
            for (int i = gTid(S); i < n; i += gThreads(S))
                x[i] += alpha * ph[i];
            gSync(S);
            o.iterations = it + 1;
            o.finalRes = sn / r0n;
            o.converged = true;
            return o;
        }
        double a3[2];
        sumOver(a3, S, rp, [&](int t0, int nt) {
            passRows<double>(A0, sh, t0, nt, [&](int i, double ti) {
                t[i] = ti;
                a3[0] += ti * ti;
                a3[1] += ti * s[i];
            });
        });
        omega = a3[0] > 1e-30 ? a3[1] / a3[0] : 0.0;
        double a4[2];
        sumOver(a4, S, rp, [&](int t0, int nt) {
            for (int i = t0; i < n; i += nt) {
                x[i] += alpha * ph[i] + omega * sh[i];
                const double ri = s[i] - omega * t[i];
                r[i] = ri;
                a4[0] += ri * ri;
                a4[1] += rh[i] * ri;
            }
        });
        o.iterations = it + 1;
        o.finalRes = sqrt(a4[0]) / r0n;
        if (o.finalRes < tol) {
            o.converged = true;
            return o;
        }
        if (fabs(omega) < 1e-30)
            break;
        rho = rhoN;
        rhoN = a4[1];
    }
    gSync(S);
    return o;
}

// r = b - A x in FP64; returns ||r||
template <int NT>
__device__ double residual(LinShared<NT> &S, int &rp, const Lv<double> &A0, const double *b,
                           const double *x, double *r) {
    double a[1];
    sumOver(a, S, rp, [&](int t0, int nt) {
        passRows<double>(A0, x, t0, nt, [&](int i, double ax) {
            const double ri = b[i] - ax;
            r[i] = ri;
            a[0] += ri * ri;
        });
    });
    return sqrt(a[0]);
}

template <int NT>
__device__ void solveOne(LinShared<NT> &S, int &rp, double *ws) {
    const DevLinSys &sys = S.sys;
    const int n = sys.n;
    const bool amg = sys.kind == kLinAmg;
    const Lv<double> A0 = levelOf<double>(sys, 0, ws + sys.lvOff);
    double *x = sys.x;
    double *r = ws;
    const double r0n = residual(S, rp, A0, sys.b, x, r);
    LinOut out{0, 0, 0.0, r0n};
    if (r0n < 1e-30) {
        out.converged = 1;
    } else if (sys.kind == kLinBicgstab) {
        const PcgOut o = bicgstab(S, rp, A0, x, ws, r0n, sys.maxIter, sys.tol);
        out.iterations = o.iterations;
        out.converged = o.converged;
        out.finalRes = o.finalRes;
    } else if (sys.precision == 0) {
        const PcgOut o = pcg<double>(S, rp, A0, x, r, ws + n, ws + 2L * n, ws + 3L * n,
                                         ws + 4L * n, ws + sys.lvOff, sys.inv, r0n, sys.maxIter,
                                         sys.tol, amg);
        out.iterations = o.iterations;
        out.converged = o.converged;
        out.finalRes = o.finalRes;
    } else {
        // mixed: FP32 PCG corrections d (A d = r) inside FP64 residual refinement
        float *f = reinterpret_cast<float *>(ws + sys.f32Off);
        float *fr = f, *fz = f + n, *fp = f + 2L * n, *fq = f + 3L * n, *ft = f + 4L * n,
              *fd = f + 5L * n;
        const Lv<float> F0 = levelOf<float>(sys, 0, f + sys.lvOff32);
        double rn = r0n;
        int total = 0;
        for (int round = 0; round < kMixedRounds && total < sys.maxIter; ++round) {
            for (int i = gTid(S); i < n; i += gThreads(S)) {
                fr[i] = float(r[i]);
                fd[i] = 0.0f;
            }
            gSync(S);
            const double innerTol = fmax(kMixedInnerTol, 0.5 * sys.tol * r0n / rn);
            const PcgOut o = pcg<float>(S, rp, F0, fd, fr, fz, fp, fq, ft, f + sys.lvOff32,
                                            sys.inv32, rn, sys.maxIter - total, innerTol, amg);
            total += o.iterations;
            for (int i = gTid(S); i < n; i += gThreads(S))
                x[i] += double(fd[i]);
            gSync(S);
            rn = residual(S, rp, A0, sys.b, x, r);
            out.finalRes = rn / r0n;
            if (out.finalRes < sys.tol) {
                out.converged = 1;
                break;
            }
            if (o.iterations == 0)
                break;
        }
        out.iterations = total;
    }
    gSync(S);
    if (gTid(S) == 0)
        *sys.out = out;
}

template <int NT>
__global__ void __launch_bounds__(NT, 1) linKernel(const DevLinSys *systems, int nsys, int *next,
                                                   double *wsBase, long wsStride) {
    __shared__ LinShared<NT> S;
    if (threadIdx.x == 0) {
        unsigned rank, ctas;
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ctas));
        S.rank = static_cast<int>(rank);
        S.ctas = static_cast<int>(ctas);
    }
    __syncthreads();
    gSync(S); // every CTA of the cluster has started: its shared memory can be written
    double *ws = wsBase + wsStride * (blockIdx.x / S.nCtas());
    int rp = 0;
    for (;;) {
        if (gTid(S) == 0) {
            const int j = atomicAdd(next, 1);
            for (int r = 0; r < S.ctas; ++r)
                putRemote(&S.job, j, r);
        }
        gSync(S);
        const int j = S.job;
        if (j >= nsys)
            break;
        {
            const int words = sizeof(DevLinSys) / 4;
            const int *src = reinterpret_cast<const int *>(systems + j);
            int *dst = reinterpret_cast<int *>(&S.sys);
            for (int t = threadIdx.x; t < words; t += NT)
                dst[t] = src[t];
        }
        __syncthreads();
        solveOne(S, rp, ws);
        gSync(S);
    }
}

} // namespace

namespace {
const void *kernelOf(const LinShape &sh) {
    return sh.threads == kLinSmallThreads ? reinterpret_cast<const void *>(&linKernel<kLinSmallThreads>)
                                          : reinterpret_cast<const void *>(&linKernel<kLinThreads>);
}
cudaError_t linConfig(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, int slots,
                      const LinShape &sh, cudaStream_t stream) {
    // the limit of the largest local levels, not of this launch: it belongs to the function, and
    // another thread may be launching it for other systems
    const void *fn = kernelOf(sh);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kLinMaxLocalBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(slots * sh.cluster);
    cfg.blockDim = dim3(sh.threads);
    cfg.dynamicSmemBytes = sh.localBytes;
    cfg.stream = stream;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = sh.cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return e;
}
} // namespace

cudaError_t launchLinear(const DevLinSys *systems, int nsys, int *next, double *ws, long wsStride,
                         int slots, const LinShape &sh, cudaStream_t stream) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cudaError_t e = linConfig(cfg, attr, slots, sh, stream);
    if (e != cudaSuccess)
        return e;
    void *args[] = {&systems, &nsys, &next, &ws, &wsStride};
    return cudaLaunchKernelExC(&cfg, kernelOf(sh), args);
}

int linConcurrent(const LinShape &sh) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    int count = 0;
    if (linConfig(cfg, attr, 1, sh, nullptr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&count, kernelOf(sh), &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return count;
}

} // namespace rq
