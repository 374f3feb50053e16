// Inner linear solvers of the small mesh classes (n <= kResCells x the CTA's threads,
// FP64 form): the recurrences of bicgstabT and pcgT (rq_solver.cu) with every vector and
// the matrix rows in registers. A group of ceil(n / 96) warps works, three cells per
// thread; only the vectors that a neighbour reads pass through shared memory. The other
// warps of the CTA join for the coarse levels of the V-cycle and wait otherwise.
//
// What bounds them: latency. One BiCGSTAB iteration is a chain of two matrix products,
// three block sums and FP64 divisions; at 384 cells the operands of all of it are 30 KB,
// so neither memory nor the FP64 pipe is near its limit. Cycles per iteration in isolation
// on a B200, by cells per thread: 384 cells 3147 / 2568 / 2677 / 3033 (1 / 2 / 3 / 4),
// 1536 cells - / - / 4916 / 5450: few warps make the block sums cheap, and four cells (11
// doubles of state each) spill out of 128 registers. With the sums on the tensor cores: 1925
// at 384 cells, 2869 at 768, 4592 at 1536. (Branch-free quotients from the approximate
// reciprocal took another 160 to 360 cycles off and were taken back: they gave NaN or zero for
// infinite, subnormal and extreme divisors. 1.4 to 6 % of a solve.)
#pragma once

// Threads of the working group, and the zero slot of an exchange vector: entries
// n .. 3T - 1 belong to no cell and hold zero, entry 3T stands for absent neighbours.
__host__ __device__ inline int resThreads(long n) {
    return static_cast<int>((n + 32 * kResCells - 1) / (32 * kResCells)) * 32;
}
// Doubles of the two exchange vectors, which start the arena; the level vectors of the
// V-cycle follow them.
__host__ __device__ inline long resExchange(long n) {
    return 2 * ((kResCells * resThreads(n) + 1L + 31) / 32 * 32);
}

extern __shared__ __align__(16) unsigned char rqSmem[];

// Sums of K values over the working group (nw warps), the same bits in every thread. A
// warp adds its lanes with two FP64 matrix products: ones times the lanes' values gives
// column sums of four lanes, of which each lane adds two and which a second product with
// ones adds up for all lanes. Five shuffle steps in their place cost 160 to 240 cycles
// (a 64-bit shuffle takes 24, 32 with 16 warps: the SM has one shuffle unit), and a
// BiCGSTAB iteration with them 2677 instead of 1925 cycles at 384 cells. The warps'
// partials are added by every thread (four at most) or once more by a product. Partials of
// warps beyond nw are zero (resClear).
template <int K> __device__ __forceinline__ void sumRes(double (&v)[K], int &rp, int nw) {
    ResShared &R = reinterpret_cast<Shared *>(rqSmem)->R;
    double u[K], w[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
        mma884(u[k], w[k], 1.0, v[k]);
#pragma unroll
    for (int k = 0; k < K; ++k)
        mma884(v[k], w[k], u[k] + w[k], 1.0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k)
            R.red[rp][k][warp] = v[k];
    groupSync(nw * 32);
    const int q = nw <= 4 ? 0 : 4 * (lane & 3);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double2 a = *reinterpret_cast<const double2 *>(&R.red[rp][k][q]);
        const double2 b = *reinterpret_cast<const double2 *>(&R.red[rp][k][q + 2]);
        v[k] = (a.x + b.x) + (a.y + b.y);
    }
    if (nw > 4)
#pragma unroll
        for (int k = 0; k < K; ++k)
            mma884(v[k], w[k], v[k], 1.0);
    rp ^= 1;
}

// Whether the square sum q passes sqrt(q) / r0n < tol: decided by q against the squared
// bound, and by the quotient itself only where rounding could matter (a square root and a
// division cost 190 cycles, twice per iteration).
__device__ __forceinline__ bool dropped(double q, double bound2, double r0n, double tol) {
    if (fabs(q - bound2) > 1e-12 * bound2)
        return q < bound2;
    return sqrt(q) / r0n < tol;
}

// A thread's rows of the 5-point system: coefficients (x neighbours in face order) and
// the exchange entries of the neighbours, packed in pairs. A row beyond n is the identity.
struct ResRows {
    double d[kResCells], a1[kResCells], a2[kResCells], aS[kResCells], aN[kResCells];
    double rd[kResCells];
    unsigned ix[kResCells], iy[kResCells];

    __device__ __forceinline__ void load(const DevClass &C, const KW<double> &K, int T) {
        const unsigned zero = kResCells * T;
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            const int c = threadIdx.x + k * T;
            d[k] = rd[k] = 1.0;
            a1[k] = a2[k] = aS[k] = aN[k] = 0.0;
            ix[k] = iy[k] = zero | (zero << 16);
            if (c < C.n) {
                const Cell q = cellOf(C, c);
                d[k] = K.d[c];
                const double w = K.aW[c], e = K.aE[c];
                a1[k] = q.xEfirst ? e : w;
                a2[k] = q.xEfirst ? w : e;
                ix[k] = static_cast<unsigned>(q.xEfirst ? q.E : q.W) |
                        (static_cast<unsigned>(q.xEfirst ? q.W : q.E) << 16);
                const unsigned s = q.south ? c - C.nx : zero, nn = q.north ? c + C.nx : zero;
                iy[k] = s | (nn << 16);
                aS[k] = q.south ? K.aS[c] : 0.0;
                aN[k] = q.north ? K.aN[c] : 0.0;
                rd[k] = (fabs(d[k]) > 1e-30) ? 1.0 / d[k] : 1.0; // jacobiPrecond as a product
            }
        }
    }
    // row k times the exchanged vector e, whose entry at the own cell is xc
    __device__ __forceinline__ double times(int k, double xc, const double *e) const {
        return d[k] * xc + a1[k] * e[ix[k] & 0xffffu] + a2[k] * e[ix[k] >> 16] +
               aS[k] * e[iy[k] & 0xffffu] + aN[k] * e[iy[k] >> 16];
    }
};

// Zero partials of absent warps and the zero slots; complete after the next group barrier.
__device__ __forceinline__ void resClear(Shared &S, double *e0, double *e1, int T) {
    for (int t = threadIdx.x; t < 2 * kResSums * kResMaxWarps; t += T)
        if ((t & (kResMaxWarps - 1)) >= T / 32)
            (&S.R.red[0][0][0])[t] = 0.0;
    if (threadIdx.x == 0)
        e0[kResCells * T] = e1[kResCells * T] = 0.0;
}

// Right-Jacobi BiCGSTAB (LinearSolver.hpp:251-345) on the rows K.d, K.aW .. K.aN;
// K.r holds b - A x0 and r0n its norm; x is updated in place. Called by the working group
// only; the caller's next CTA barrier makes x and *out visible. (s, s) is summed together
// with (t, t) and (t, s): one block sum fewer per iteration for at most one matrix product
// more per solve.
__device__ __noinline__ void bicgstabRes(double *x, double r0n, int maxIter, double tol,
                                         LinRes *out) {
    Shared &S = *reinterpret_cast<Shared *>(rqSmem);
    const DevClass &C = S.C;
    const int n = C.n, nw = S.resWarps, T = nw * 32;
    double *e0 = reinterpret_cast<double *>(rqSmem + kSharedBytes);
    double *e1 = e0 + resExchange(n) / 2;
    LinRes res{0, 0.0, r0n, false};
    if (r0n < 1e-30) {
        res.converged = true;
        if (threadIdx.x == 0)
            *out = res;
        return;
    }
    ResRows A;
    double r[kResCells], rh[kResCells], p[kResCells], v[kResCells], xv[kResCells];
    A.load(C, S.K64, T);
    double acc[1] = {0.0};
#pragma unroll
    for (int k = 0; k < kResCells; ++k) {
        const int c = threadIdx.x + k * T;
        p[k] = v[k] = 0.0;
        r[k] = c < n ? S.K64.r[c] : 0.0;
        xv[k] = c < n ? x[c] : 0.0;
        rh[k] = r[k];
        acc[0] += r[k] * r[k];
    }
    resClear(S, e0, e1, T);
    int rp = 0;
    sumRes<1>(acc, rp, nw);
    const double bound2 = (tol * r0n) * (tol * r0n);
    double rhoN = acc[0], rho = 1, alphaOm = 1, omega = 1;
    double last = r0n * r0n;
    for (int it = 0; it < maxIter; ++it) {
        if (fabs(rhoN) < 1e-30)
            break;
        const double beta = (rhoN / (rho + 1e-30)) * alphaOm;
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            p[k] = r[k] + beta * (p[k] - omega * v[k]);
            e0[threadIdx.x + k * T] = p[k] * A.rd[k];
        }
        groupSync(T);
        double s1[1] = {0.0};
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            v[k] = A.times(k, p[k] * A.rd[k], e0);
            s1[0] += rh[k] * v[k];
        }
        sumRes<1>(s1, rp, nw);
        if (fabs(s1[0]) < 1e-30)
            break;
        const double alpha = rhoN / s1[0];
        double s3[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < kResCells; ++k) { // r holds s until the iteration's end
            r[k] -= alpha * v[k];
            e1[threadIdx.x + k * T] = r[k] * A.rd[k];
            s3[2] += r[k] * r[k];
        }
        groupSync(T);
        double t[kResCells];
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            t[k] = A.times(k, r[k] * A.rd[k], e1);
            s3[0] += t[k] * t[k];
            s3[1] += t[k] * r[k];
        }
        sumRes<3>(s3, rp, nw);
        res.iterations = it + 1;
        last = s3[2];
        if (dropped(s3[2], bound2, r0n, tol)) {
#pragma unroll
            for (int k = 0; k < kResCells; ++k)
                xv[k] += alpha * (p[k] * A.rd[k]);
            res.converged = true;
            break;
        }
        omega = (s3[0] > 1e-30) ? s3[1] / s3[0] : 0.0;
        double s4[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            xv[k] += alpha * (p[k] * A.rd[k]) + omega * (r[k] * A.rd[k]);
            r[k] -= omega * t[k];
            s4[0] += r[k] * r[k];
            s4[1] += rh[k] * r[k];
        }
        alphaOm = alpha / (omega + 1e-30);
        sumRes<2>(s4, rp, nw);
        last = s4[0];
        if (dropped(s4[0], bound2, r0n, tol)) {
            res.converged = true;
            break;
        }
        if (fabs(omega) < 1e-30)
            break;
        rho = rhoN;
        rhoN = s4[1];
    }
#pragma unroll
    for (int k = 0; k < kResCells; ++k) {
        const int c = threadIdx.x + k * T;
        if (c < n)
            x[c] = xv[k];
    }
    if (threadIdx.x == 0) {
        res.finalRes = sqrt(last) / r0n;
        *out = res;
    }
}

__device__ __forceinline__ int up32(int n) { return (n + 31) & ~31; }

// Levels of the V-cycle (thread 0, from carve): vectors, operator
// values where the refresh writes them, and the constant tables and the coarsest inverse
// in the arena as far as place() finds room, in the order of their use per byte.
template <typename Place> __device__ void resPlace(Shared &S, Place place) {
    const DevClass &C = S.C;
    const int L = C.nlev;
    for (int l = 0; l < L; ++l) {
        const DevAmgLevel &F = C.lev[l];
        ResLevel &R = S.RL[l];
        double *v = localLevel(S, l) ? levelVec<double>(S, S.K64, l) : S.W.amgVec + F.vecOff;
        R.n = F.n;
        R.sh = 0;
        while (R.sh < 5 && (2 << R.sh) * F.n <= static_cast<int>(blockDim.x) &&
               (2 << R.sh) <= F.n)
            ++R.sh;
        R.vOff = static_cast<int>(reinterpret_cast<unsigned char *>(v) - rqSmem);
        R.b = v;
        R.xa = v + F.n;
        R.x = v + 2 * F.n;
        R.r = v + 3 * F.n;
        R.rd = v + 4 * F.n;
        R.aw = F.width;
        R.av = S.W.amgVal + F.valOff;
        R.ac = F.ecol16;
        R.pw = l + 1 < L ? F.pw : 0;
        R.pc = F.pcol16;
        R.pv = F.pval;
        R.rw = l > 0 ? C.lev[l - 1].rw : 0;
        R.rc = l > 0 ? C.lev[l - 1].rcol16 : nullptr;
        R.rv = l > 0 ? C.lev[l - 1].rval : nullptr;
    }
    auto put16 = [&](const uint16_t *&p, int cnt) {
        if (double *q = place((cnt + 3) / 4))
            p = reinterpret_cast<const uint16_t *>(q);
    };
    auto put = [&](const double *&p, int cnt) {
        if (double *q = place(cnt))
            p = q;
    };
    // a cluster's CTAs place the levels they run whole, with copies of the operator values
    const int first = kCluster ? C.locLevel : 0;
    for (int l = L - 2; l >= 1 && l >= first; --l) {
        ResLevel &R = S.RL[l];
        put16(R.ac, R.aw * up32(R.n));
        if (kCluster)
            put(R.av, R.aw * up32(R.n));
    }
    for (int l = L - 1; l >= first; --l) {
        ResLevel &R = S.RL[l];
        if (l > 0) {
            put16(R.rc, R.rw * up32(R.n));
            put(R.rv, R.rw * up32(R.n));
        }
        if (l + 1 < L) {
            put16(R.pc, R.pw * up32(R.n));
            put(R.pv, R.pw * up32(R.n));
        }
    }
    const int m = S.RL[L - 1].n, seg = 1 << S.RL[L - 1].sh;
    S.resInv = place(static_cast<long>((m + seg - 1) / seg) * m * seg);
    S.ownInv = S.resInv != nullptr;
}

// Copies the constant tables that resPlace put into the arena (all threads).
__device__ __noinline__ void resTables(Shared &S) {
    const DevClass &C = S.C;
    const int L = C.nlev, t0 = threadIdx.x, ts = blockDim.x;
    auto copy = [&](auto *dst, const auto *src, int cnt) {
        if (dst != src)
            for (int e = t0; e < cnt; e += ts)
                const_cast<std::remove_const_t<std::remove_reference_t<decltype(*dst)>> *>(dst)[e] =
                    src[e];
    };
    for (int l = 0; l < L; ++l) {
        const ResLevel &R = S.RL[l];
        const DevAmgLevel &F = C.lev[l];
        if (l > 0 && l + 1 < L)
            copy(R.ac, F.ecol16, R.aw * up32(R.n));
        if (l + 1 < L) {
            copy(R.pc, F.pcol16, R.pw * up32(R.n));
            copy(R.pv, F.pval, R.pw * up32(R.n));
        }
        if (l > 0) {
            copy(R.rc, C.lev[l - 1].rcol16, R.rw * up32(R.n));
            copy(R.rv, C.lev[l - 1].rval, R.rw * up32(R.n));
        }
    }
    __syncthreads();
}

// After a refresh: the inverse of the coarsest level in the order in which coarseRes reads
// it (entry u * (m seg) + t is row t / seg, column t % seg + u seg), and a cluster's copies
// of the operator values.
__device__ __noinline__ void denseOrder(Shared &S) {
    const DevClass &C = S.C;
    if (S.ownInv || ctaRank() == 0) {
        const ResLevel &R = S.RL[C.nlev - 1];
        const int m = R.n, seg = 1 << R.sh, w = m * seg;
        const double *inv = m <= 32 ? S.coarse : S.W.dense0 + m;
        const int ld = m <= 32 ? m : 2 * m;
        for (int e = threadIdx.x; e < (m + seg - 1) / seg * w; e += blockDim.x) {
            const int u = e / w, t = e - u * w, i = t >> R.sh, k = t - (i << R.sh) + u * seg;
            if (k < m)
                S.resInv[e] = inv[i * ld + k];
        }
    }
    if constexpr (kCluster)
        for (int l = C.locLevel; l + 1 < C.nlev; ++l) {
            const ResLevel &R = S.RL[l];
            const double *from = S.W.amgVal + C.lev[l].valOff;
            double *to = const_cast<double *>(R.av);
            if (to != from)
                for (int e = threadIdx.x; e < R.aw * up32(R.n); e += blockDim.x)
                    to[e] = from[e];
        }
    SYNC();
}

// One row of an ELL table (16-bit columns) times the gathered vector; padding
// entries have value 0 and column 0. Columns and values of up to eleven entries are loaded
// before the first of them is used.
template <int W>
__device__ __forceinline__ double rowFix(const uint16_t *cols, const double *val,
                                         const double *vec) {
    constexpr int B = W <= 11 ? W : 8;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 0; k < W; k += B) {
        unsigned c[B];
        double v[B];
#pragma unroll
        for (int u = 0; u < B && k + u < W; ++u) {
            c[u] = cols[32 * (k + u)];
            v[u] = val[32 * (k + u)];
        }
#pragma unroll
        for (int u = 0; u < B && k + u < W; ++u)
            (u & 1 ? s1 : s0) += v[u] * vec[c[u]];
    }
    return s0 + s1;
}
// The usual widths (channels of 3 to 5 cells: 2, 4, 11, 15; bump meshes: 1, 4, 9, 11) get
// code of their own: a phase of the V-cycle is bound by the instructions it issues, and a
// loop with a run-time width and bounds checks takes 5 times as many (1600 cycles for 192
// rows of 11 entries).
__device__ __forceinline__ double rowRes(const uint16_t *cols, const double *val,
                                         const double *vec, int width, int row) {
    cols += ellRow(row, width);
    val += ellRow(row, width);
    switch (width) {
    case 1: return rowFix<1>(cols, val, vec);
    case 2: return rowFix<2>(cols, val, vec);
    case 4: return rowFix<4>(cols, val, vec);
    case 9: return rowFix<9>(cols, val, vec);
    case 11: return rowFix<11>(cols, val, vec);
    case 15: return rowFix<15>(cols, val, vec);
    default: break;
    }
    double s = 0.0;
    int k = 0;
    for (; k + 4 <= width; k += 4)
        s += rowFix<4>(cols + 32 * k, val + 32 * k, vec);
    for (; k < width; ++k)
        s += val[32 * k] * vec[cols[32 * k]];
    return s;
}

// The coarse levels of one V-cycle (vcycleT): the level-0 residual in rr0 is restricted,
// and level 1's solution is left in its x. All threads take part (levelThreads); the
// caller's barrier precedes.
// With Resident the vectors are known to be in shared memory (and loaded as such: 32-bit
// addresses).
template <bool Resident> __device__ __forceinline__ ResLevel levelOf(const Shared &S, int l) {
    ResLevel R = S.RL[l];
    if constexpr (Resident) {
        double *v = reinterpret_cast<double *>(rqSmem + R.vOff);
        R.b = v;
        R.xa = v + R.n;
        R.x = v + 2 * R.n;
        R.r = v + 3 * R.n;
        R.rd = v + 4 * R.n;
    }
    return R;
}
// out = x + om (b - A x) / diag on level l
template <bool SH>
__device__ __forceinline__ void smoothRes(const Shared &S, int l, const ResLevel &R,
                                          const double *x, double *out) {
    const double om = S.C.amgW;
    const int ts = levelThreads(S, l);
    for (int i = levelTid(S, l); i < R.n; i += ts)
        out[i] = x[i] + om * (R.b[i] - rowRes(R.ac, R.av, x, R.aw, i)) * R.rd[i];
    levelSync(S, l);
}
// level l on the way down: right-hand side from the residual fr above, pre-smoothing from
// zero, residual
template <bool SH>
__device__ __forceinline__ void downRes(const Shared &S, int l, const double *fr) {
    const ResLevel R = levelOf<SH>(S, l);
    const bool two = S.C.amgSweeps >= 2;
    const double om = S.C.amgW;
    const int t0 = levelTid(S, l), ts = levelThreads(S, l);
    for (int i = t0; i < R.n; i += ts) {
        const double bi = rowRes(R.rc, R.rv, fr, R.rw, i);
        R.b[i] = bi;
        R.xa[i] = om * bi * R.rd[i];
    }
    levelSync(S, l);
    if (two)
        smoothRes<SH>(S, l, R, R.xa, R.x);
    const double *x = two ? R.x : R.xa;
    for (int i = t0; i < R.n; i += ts)
        R.r[i] = R.b[i] - rowRes(R.ac, R.av, x, R.aw, i);
    levelSync(S, l);
}
// and on the way up: the correction xc of the level below, post-smoothing; the solution in x.
// The corrected iterate replaces the pre-smoothed one, each thread its own rows. It must not go
// to r: on a cluster the level below restricts this level's r in every CTA, with no cluster
// barrier since, and a CTA that is late would read iterates for residuals.
template <bool SH>
__device__ __forceinline__ void upRes(const Shared &S, int l, const double *xc) {
    const ResLevel R = levelOf<SH>(S, l);
    const bool two = S.C.amgSweeps >= 2;
    const double al = S.C.amgAlpha;
    double *x = two ? R.x : R.xa;
    const int ts = levelThreads(S, l);
    for (int i = levelTid(S, l); i < R.n; i += ts)
        x[i] += al * rowRes(R.pc, R.pv, xc, R.pw, i);
    levelSync(S, l);
    smoothRes<SH>(S, l, R, x, two ? R.xa : R.x);
    if (two)
        smoothRes<SH>(S, l, R, R.xa, R.x);
}
// levels l0 .. L - 1, all with vectors in shared memory (SH) or wherever they are
template <bool SH>
__device__ __forceinline__ void levelsRes(Shared &S, int l0, const double *fr) {
    const int L = S.C.nlev;
    for (int l = l0; l + 1 < L; ++l) {
        downRes<SH>(S, l, fr);
        fr = levelOf<SH>(S, l).r;
    }
    const int l = L - 1;
    const ResLevel R = levelOf<SH>(S, l);
    const int t0 = levelTid(S, l), ts = levelThreads(S, l);
    for (int i = t0; i < R.n; i += ts)
        R.b[i] = L == 1 ? fr[i] : rowRes(R.rc, R.rv, fr, R.rw, i);
    levelSync(S, l);
    // 1 << sh threads per row of the dense inverse
    const int seg = 1 << R.sh, w = R.n << R.sh, j = t0 & (seg - 1);
    for (int base = 0; base < w; base += ts) {
        const int t = base + t0;
        double s0 = 0.0, s1 = 0.0;
        if (t < w) {
            const double *q = S.resInv + t, *v = R.b + j;
            int k = j;
            for (; k + 7 * seg < R.n; k += 8 * seg, q += 8 * w, v += 8 * seg) {
                double a[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    a[u] = q[u * w];
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    s0 += a[u] * v[u * seg];
                    s1 += a[u + 1] * v[(u + 1) * seg];
                }
            }
            for (; k < R.n; k += seg, q += w, v += seg)
                s0 += q[0] * v[0];
        }
        s0 += s1;
        for (int o = seg >> 1; o > 0; o >>= 1)
            s0 += __shfl_xor_sync(FULL, s0, o);
        if (j == 0 && t < w)
            R.x[t >> R.sh] = s0;
    }
    levelSync(S, l);
    for (int k = L - 2; k >= l0; --k)
        upRes<SH>(S, k, levelOf<SH>(S, k + 1).x);
}
// rr0: the level-0 residual
template <bool Resident>
__device__ __forceinline__ void coarseRes(Shared &S, const double *rr0) {
    if constexpr (kCluster) {
        const int loc = S.C.locLevel;
        const double *fr = rr0;
        for (int l = 1; l < loc; ++l) {
            downRes<false>(S, l, fr);
            fr = S.RL[l].r;
        }
        levelsRes<true>(S, loc, fr);
        for (int l = loc - 1; l >= 1; --l)
            upRes<false>(S, l, S.RL[l + 1].x);
    } else {
        levelsRes<Resident>(S, S.C.nlev > 1 ? 1 : 0, rr0);
    }
}

// PCG (LinearSolver.hpp:184-246 / :908-982) from x = 0 (set by the assembly), with the V-cycle or the Jacobi
// preconditioner; K64.r holds b and r0n its norm. The working group
// holds the finest level in registers; all threads of the CTA run the coarse levels. The
// caller's next CTA barrier makes x and *out visible.
// What bounds it: the instructions that each of its 13 to 21 phases issues. Measured on a
// B200, us of the pressure solve per PCG iteration (the first 400 outer iterations): 8.0 / 15.4 /
// 25.3 at 384 / 768 / 1536 cells, against 12.2 / 27.2 / 48.3 of pcgT and vcycleT before.
template <bool AMG>
__device__ __noinline__ void pcgRes(double *x, double r0n, int maxIter, double tol, LinRes *out) {
    Shared &S = *reinterpret_cast<Shared *>(rqSmem);
    const DevClass &C = S.C;
    const int n = C.n, nw = S.resWarps, T = nw * 32;
    double *e0 = reinterpret_cast<double *>(rqSmem + kSharedBytes);
    double *e1 = e0 + resExchange(n) / 2;
    LinRes res{0, 0.0, r0n, false};
    const bool mine = static_cast<int>(threadIdx.x) < T;
    if (r0n < 1e-30) {
        res.converged = true;
        if (threadIdx.x == 0)
            *out = res;
        return;
    }
    const int L = C.nlev;
    const bool two = AMG && C.amgSweeps >= 2;
    const double om = C.amgW, al = C.amgAlpha;
    const double bound2 = (tol * r0n) * (tol * r0n);
    ResRows A;
    double r[kResCells], p[kResCells];
    int rp = 0;
    double rz = 0.0;
    if (mine) {
        A.load(C, S.K64, T);
#pragma unroll
        for (int k = 0; k < kResCells; ++k) {
            const int c = threadIdx.x + k * T;
            r[k] = c < n ? S.K64.r[c] : 0.0;
            p[k] = 0.0;
        }
        resClear(S, e0, e1, T);
    }
    for (int it = 0;; ++it) {
        double z[kResCells], q[1] = {0.0};
        if constexpr (AMG) {
            if (mine && L > 1) { // pre-smoothed iterate in e0, the residual in e1
                double *first = two ? e1 : e0;
#pragma unroll
                for (int k = 0; k < kResCells; ++k)
                    first[threadIdx.x + k * T] = om * r[k] * A.rd[k];
                groupSync(T);
                if (two) {
#pragma unroll
                    for (int k = 0; k < kResCells; ++k) {
                        const double z0 = om * r[k] * A.rd[k];
                        e0[threadIdx.x + k * T] = z0 + om * (r[k] - A.times(k, z0, e1)) * A.rd[k];
                    }
                    groupSync(T);
                }
#pragma unroll
                for (int k = 0; k < kResCells; ++k)
                    e1[threadIdx.x + k * T] = r[k] - A.times(k, e0[threadIdx.x + k * T], e0);
            } else if (mine) {
#pragma unroll
                for (int k = 0; k < kResCells; ++k)
                    e1[threadIdx.x + k * T] = r[k];
            }
            __syncthreads();
            coarseRes<true>(S, e1);
        }
        if (mine) {
            if (AMG && L > 1) {
                const ResLevel &R = S.RL[0];
                const double *xc = levelOf<true>(S, 1).x;
                double pz[kResCells];
#pragma unroll
                for (int k = 0; k < kResCells; ++k) {
                    const int c = threadIdx.x + k * T;
                    pz[k] = c < n ? rowRes(R.pc, R.pv, xc, R.pw, c) : 0.0;
                }
#pragma unroll
                for (int k = 0; k < kResCells; ++k) {
                    z[k] = e0[threadIdx.x + k * T] + al * pz[k];
                    e0[threadIdx.x + k * T] = z[k];
                }
                groupSync(T);
                if (two) {
#pragma unroll
                    for (int k = 0; k < kResCells; ++k) {
                        z[k] += om * (r[k] - A.times(k, z[k], e0)) * A.rd[k];
                        e1[threadIdx.x + k * T] = z[k];
                    }
                    groupSync(T);
                }
                const double *e = two ? e1 : e0;
#pragma unroll
                for (int k = 0; k < kResCells; ++k) {
                    z[k] += om * (r[k] - A.times(k, z[k], e)) * A.rd[k];
                    q[0] += r[k] * z[k];
                }
            } else {
#pragma unroll
                for (int k = 0; k < kResCells; ++k) {
                    const int c = threadIdx.x + k * T;
                    z[k] = AMG ? (c < n ? S.RL[0].x[c] : 0.0) : r[k] * A.rd[k];
                    q[0] += r[k] * z[k];
                }
            }
            sumRes<1>(q, rp, nw);
            const double beta = it == 0 ? 0.0 : q[0] / (rz + 1e-30);
            rz = q[0];
            q[0] = 0.0;
#pragma unroll
            for (int k = 0; k < kResCells; ++k) {
                p[k] = z[k] + beta * p[k];
                e1[threadIdx.x + k * T] = p[k];
            }
            groupSync(T);
            double Ap[kResCells];
#pragma unroll
            for (int k = 0; k < kResCells; ++k) {
                Ap[k] = A.times(k, p[k], e1);
                q[0] += p[k] * Ap[k];
            }
            sumRes<1>(q, rp, nw);
            bool done = false;
            if (fabs(q[0]) < 1e-30) {
                res.breakdown = true;
                done = true;
            } else {
                const double alpha = rz / q[0];
                q[0] = 0.0;
#pragma unroll
                for (int k = 0; k < kResCells; ++k) {
                    const int c = threadIdx.x + k * T;
                    r[k] -= alpha * Ap[k];
                    q[0] += r[k] * r[k];
                    if (c < n)
                        x[c] += alpha * p[k];
                }
                sumRes<1>(q, rp, nw);
                res.iterations = it + 1;
                res.finalRes = q[0]; // its square until the end
                res.converged = dropped(q[0], bound2, r0n, tol);
                done = res.converged || it + 1 >= maxIter;
            }
            if (threadIdx.x == 0)
                S.resDone = done;
            if (!AMG && done)
                break;
        }
        if constexpr (AMG) {
            __syncthreads();
            if (S.resDone)
                break;
        } else if (!mine) {
            break;
        }
    }
    if (threadIdx.x == 0) {
        res.finalRes = sqrt(res.finalRes) / r0n;
        *out = res;
    }
}
