// The B200 forward model: one CTA (a thread-block cluster for large meshes) runs one
// SIMPLE + k-omega SST solve, every outer iteration of it, from cold start to its verdict, with all state in
// HBM/L2 and the CTA's shared memory. Persistent CTAs pull draws from a job
// queue (atomic counter), so a batch of mixed mesh classes keeps every SM busy
// until the longest solve ends; a serving loop launches the same kernel per
// admitted request on its own stream.
//
// The loop restates SIMPLESolver::solve (rans-uq/src/SIMPLESolver.cpp:1193-1716)
// on the structured periodic layout of rq_setup.h. Every face sum is gathered
// per cell; dot products are block reductions (FP64 matrix products add a warp's
// lanes, then shuffles the warp partials, which every
// thread evaluates identically, so control flow stays uniform in the CTA).
//
// Inner solvers (core/include/LinearSolver.hpp): right-Jacobi BiCGSTAB
// (:251-345) for momentum, k and omega; for the pressure correction PCG
// (:184-246) with Jacobi or with the AMG V-cycle of this project (fixed
// aggregation from rq_setup.cpp, damped-Jacobi smoothing, Galerkin values
// refreshed when it degrades, dense coarsest inverse), or BiCGSTAB. Classes of up to
// 1536 cells run them in registers (rq_resident.cuh).
#include "rq_device.cuh"
#include "rq_kernels.h"

#include <cuda_runtime.h>
#include <math.h>

#include <type_traits>

namespace rq {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// A solve runs on one CTA, or (objects compiled with RQ_CLUSTER) on a thread-block cluster
// of 1 to 8 CTAs, which share the workspace in global memory: cells, faces and rows are dealt
// out over all threads of the cluster, SYNC is its barrier, and block sums end in an exchange
// of partial sums through distributed shared memory. Each CTA keeps its own copy of the
// shared-memory state (Shared) and derives the same values in it. A class's sums are formed
// in a fixed number of slices (solveSlices), of which a CTA holds one or several, so the
// number of CTAs changes no bit of a result.
#ifdef RQ_CLUSTER
constexpr bool kCluster = true;
#else
constexpr bool kCluster = false;
#endif
__device__ __forceinline__ int ctaRank() {
    unsigned r = 0;
    if constexpr (kCluster)
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return static_cast<int>(r);
}
__device__ __forceinline__ int ctaCount() {
    unsigned r = 1;
    if constexpr (kCluster)
        asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
    return static_cast<int>(r);
}
__device__ __forceinline__ int gTid() { return ctaRank() * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int gThreads() { return ctaCount() * blockDim.x; }
__device__ __forceinline__ void SYNC() {
    if (kCluster && ctaCount() > 1)
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    else
        __syncthreads();
}
// stores v at the address that p has in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ void putRemote(double *p, double v, int rank) {
    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\t"
                 "st.shared::cluster.f64 [r], %2;\n\t}" ::"r"(a), "r"(rank), "d"(v) : "memory");
}
__device__ __forceinline__ void putRemote(int *p, int v, int rank) {
    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\t"
                 "st.shared::cluster.s32 [r], %2;\n\t}" ::"r"(a), "r"(rank), "r"(v) : "memory");
}
constexpr int kRedSlots = 8; // values per block reduction
constexpr int kSumSlots = 3; // of a sum
// rows of warp partials: a reduction's values, or a sum's of every slice that a CTA holds
constexpr int kRedRows = kCluster ? kMaxSlices * kSumSlots : kRedSlots;
constexpr int kRedWarps = kCluster ? 24 : 32; // the cluster kernels' CTAs have 24 warps
#ifdef RQ_CLUSTER
static_assert(RQ_CTA == 32 * kRedWarps, "a column per warp");
#endif

struct Work {
    double *Ux, *Uy, *p, *k, *w, *nuT, *F1, *F2, *Pk, *CD, *S;
    double *gUxx, *gUxy, *gUyx, *gUyy, *gKx, *gKy, *gWx, *gWy, *gPx, *gPy;
    double *phi, *phiPred, *pCoeff; // x faces [0,n) then y faces [n, n+nfy)
    double *fScr;                            // face scratch of the transport assemblies
    double *d, *aW, *aE, *aS, *aN, *b, *aP; // aP: V / a_P of the x momentum rows
    double *Uxp, *Uyp, *kOld, *wOld, *pp;
    double *r, *rh, *pv, *v, *s, *t, *ph, *sh;
    double *z, *xa, *xb, *rr;                // PCG / level-0 V-cycle
    double *rd;                              // reciprocal diagonal of the system being solved
    double *amgVal, *amgVec, *dense0, *dense1;
};

// Krylov / AMG storage of one value type (see "inner linear solvers").
template <typename T> struct KW {
    T *d, *aW, *aE, *aS, *aN, *rd;        // matrix and reciprocal diagonal
    T *r, *rh, *pv, *v, *s, *t, *ph, *sh; // BiCGSTAB
    T *z, *xa, *xb, *rr;                  // PCG / level-0 V-cycle (share BiCGSTAB-only storage)
    T *x;                                 // FP32 correction of the mixed form
    T *amgVal, *amgVec;                   // coarse levels: values; b, xa, xb, r, 1/diag
};

struct LinRes {
    int iterations;
    double finalRes, initialRes;
    bool converged;
    bool breakdown = false; // stopped on the |p.Ap| < 1e-30 guard (a round-off right-hand side)
};

// The outer loop's scalars. Every thread derives them identically from the same
// block reductions and writes the same value, so they can live here rather than in
// registers: a phase call then has no live loop state to save and restore around it
// (those saves were local-memory traffic that missed L1 at large meshes).
struct LoopState {
    double lastK, lastW, worst, fluxRef, n0x, n0y, n0p, rateU;
    double momRes, momScale, contScaled, fluxScale, uChange;
    LinRes resU[2], resP, resK, resW;
    int amgNeed, amgAfter, status, finalIter;
    bool established, converged, diverged;
};

// Shared memory of the resident solvers (rq_resident.cuh): block sums in alternating
// buffers, up to three values of up to 16 warps.
constexpr int kResCells = 3;        // cells per thread
constexpr int kResMaxThreads = 512; // CTA size up to which a thread has 128 registers
constexpr int kResMaxWarps = 16;
constexpr int kResSums = 3;
struct alignas(16) ResShared {
    double red[2][kResSums][kResMaxWarps];
};

// One level of the FP64 V-cycle (coarseRes): its rows, the threads per row of the dense
// coarsest solve (1 << sh), its operator, the prolongation to it from the next level and
// the restriction of the level above (widths, 16-bit columns and values in ELL form), and
// its vectors: right-hand side, iterate, solution, residual, 1/diag.
struct ResLevel {
    int n, sh, aw, pw, rw, vOff; // vOff: byte offset of the vectors in shared memory
    const uint16_t *ac, *pc, *rc;
    const double *av, *pv, *rv;
    double *b, *xa, *x, *r;
    const double *rd;
};

struct Shared {
    DevClass C;
    Work W;
    KW<double> K64;
    KW<float> K32;
    double coeff[11];
    alignas(16) double red[2][kRedRows][kRedWarps];
    double cred[2][kRedSlots][kCluster ? kMaxSlices : 1]; // sums of the cluster's slices
    int slices, ownSlices; // of the class's sums, and of these the CTA's
    double ring[4][kWindowCap];  // U, k, omega, Q change samples
    int cnt[4];
    double q[kMaxProbes], qPrev[kMaxProbes];
    int haveQPrev;
    int job;
    DevJob jd; // the request being served (a copy out of host-mapped memory)
    int admitted;
    long long innerKrylov, innerPressure; // inner iterations of the solve (work accounting)
    long long stage[8];                   // clock64 cycles per stage (thread 0)
    long long tmark;
    double wallBeta;  // beta1 the wall-face omega was last set with (applyAllBCs' default
                      // on a cold start, the cached solve's on a warm one, then b1)
    double coarse[32 * 32];               // in-place inverse of a coarsest level of <= 32 rows
    LoopState L;                          // the outer loop's scalars (runSolve)
    ResShared R;                          // block sums of the resident solvers
    int resWarps;                         // their working warps, 0: the general solvers
    int resAmg;                           // the V-cycle too
    double *resInv;                       // the coarsest inverse in coarseRes's order,
    int ownInv;                           // a CTA's own copy in shared memory
    int resDone;                          // a PCG solve has ended
    ResLevel RL[kMaxLevels];              // levels of the FP64 V-cycle, filled where lean is set
    int lean;                             // coarseRes runs the coarse levels
    double *locVec;                       // vectors of a cluster's CTA-local levels
};

// dynamic shared memory of every solve kernel: Shared, then the arena
constexpr size_t kSharedBytes = (sizeof(Shared) + 15) / 16 * 16;

// stage timers, as the reference's momentum / pressure / turbulence timers
// (rans-uq/include/SIMPLESolver.hpp:293-305): 0 set-up, 1 closure, 2 momentum,
// 3 pressure assembly, 4 pressure solve, 5 AMG refresh, 6 turbulence, 7 bookkeeping
__device__ __forceinline__ void mark(Shared &S, int k) {
    if (threadIdx.x == 0) {
        const long long t = clock64();
        S.stage[k] += t - S.tmark;
        S.tmark = t;
    }
}

// barrier of the CTA's first `threads` threads (a multiple of 32)
__device__ __forceinline__ void groupSync(int threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// ---------------------------------------------------------------- reductions
// D = A B of one FP64 m8n8k4 product: a is this lane's A[lane / 4][lane % 4], b its
// B[lane % 4][lane / 4]; d0, d1 receive D[lane / 4][2 (lane % 4) + 0, 1].
__device__ __forceinline__ void mma884(double &d0, double &d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};"
        : "=d"(d0), "=d"(d1)
        : "d"(a), "d"(b), "d"(0.0));
}

// Block reductions. A warp adds its lanes with two FP64 matrix products (sumRes); lane 0
// parks the sum in shared memory, and after one barrier every warp adds the same partials
// by the same shuffles -- so all threads of the CTA hold bit-identical values and branch
// alike. (With matrix products for the partials too, which every warp repeats, the solves of
// the general solvers took 8 to 14 % longer: mixed form, 384 / 768 / 1536 cells 166 / 286 / 448
// us per outer iteration against 146 / 264 / 416; with shuffles for both 152 / 271 / 425.)
//
// Slice i of `slices` holds the cells (i + k slices) blockDim + 0 .. blockDim - 1, k = 0, 1, ...
// CTA r of c CTAs holds the slices r, r + c, ..., which are the cells of its own sweeps
// (FOR_OWN). Within a slice a thread adds its cells, a warp its threads and the slice its
// warps, whichever CTA does it, and every thread adds the slices in order.
template <int K>
__device__ __forceinline__ void parkSums(double (&v)[K], Shared &S, int rp, int slice) {
    static_assert(K <= kSumSlots, "rows of a slice's sums");
    double u[K], w[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
        mma884(u[k], w[k], 1.0, v[k]);
#pragma unroll
    for (int k = 0; k < K; ++k)
        mma884(v[k], w[k], u[k] + w[k], 1.0);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < K; ++k)
            S.red[rp][slice * K + k][threadIdx.x >> 5] = v[k];
}
__device__ __forceinline__ double addLanes(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    return v;
}
// the sums of the parked partials, in every thread; a barrier for what was stored before
template <int K>
__device__ __forceinline__ void totalSums(double (&v)[K], Shared &S, int &rp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if constexpr (kCluster) { // a warp per slice and value, the sums to every CTA
        const int nc = ctaCount(), rank = ctaRank(), rows = S.ownSlices * K;
        for (int t = warp; t < rows; t += nw) {
            double w = 0.0, unused; // eight partials per lane, four lanes by a product: one warp
                                    // does it, so it costs less than five shuffles here
            if (8 * (lane & 3) < nw) {
                const double2 *r = reinterpret_cast<const double2 *>(&S.red[rp][t][8 * (lane & 3)]);
                const double2 a = r[0], b = r[1], c = r[2], d = r[3];
                w = ((a.x + b.x) + (c.x + d.x)) + ((a.y + b.y) + (c.y + d.y));
            }
            mma884(w, unused, w, 1.0);
            const int slice = t / K, k = t - slice * K;
            if (lane < nc)
                putRemote(&S.cred[rp][k][slice * nc + rank], w, lane);
        }
        SYNC();
        const int ns = S.slices;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = S.cred[rp][k][0];
            for (int c = 1; c < ns; ++c)
                v[k] += S.cred[rp][k][c];
        }
    } else { // every warp the same partials
#pragma unroll
        for (int k = 0; k < K; ++k)
            v[k] = addLanes(lane < nw ? S.red[rp][k][lane] : 0.0);
    }
    rp ^= 1;
}
// add(i) adds item i's terms to v, for the thread's items of 0 .. count - 1; one value of v
// per slice is parked
template <int K, typename Add>
__device__ __forceinline__ void parkOver(double (&v)[K], Shared &S, int rp, int count, Add add) {
    const int own = kCluster ? S.ownSlices : 1;
    const int step = (kCluster ? S.slices : 1) * blockDim.x;
    for (int slice = 0; slice < own; ++slice) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            v[k] = 0.0;
        for (int i = (slice * ctaCount() + ctaRank()) * blockDim.x + threadIdx.x; i < count; i += step)
            add(i);
        parkSums(v, S, rp, slice);
    }
}
template <int K, typename Add>
__device__ __forceinline__ void sumOver(double (&v)[K], Shared &S, int &rp, int count, Add add) {
    parkOver(v, S, rp, count, add);
    totalSums(v, S, rp);
}

// Maximum over a warp of nonnegative values: their bit patterns are ordered as integers, so
// the high words' maximum and then the low words' among its holders (two reductions in place
// of ten shuffles).
__device__ __forceinline__ double warpMax(double v) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v));
    const unsigned mh = __reduce_max_sync(FULL, hi);
    const unsigned ml =
        __reduce_max_sync(FULL, hi == mh ? static_cast<unsigned>(__double2loint(v)) : 0u);
    return __hiloint2double(static_cast<int>(mh), static_cast<int>(ml));
}
// Maxima of K nonnegative values over the block.
template <int K>
__device__ __forceinline__ void blockMax(double (&v)[K], Shared &S, int &rp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
        v[k] = warpMax(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k)
            S.red[rp][k][warp] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k)
        v[k] = warpMax(lane < nw ? S.red[rp][k][lane] : 0.0);
    if constexpr (kCluster) {
        const int nc = ctaCount(), rank = ctaRank();
        if (static_cast<int>(threadIdx.x) < nc)
#pragma unroll
            for (int k = 0; k < K; ++k)
                putRemote(&S.cred[rp][k][rank], v[k], threadIdx.x);
        SYNC();
#pragma unroll
        for (int k = 0; k < K; ++k)
            for (int c = 0; c < nc; ++c)
                v[k] = fmax(v[k], S.cred[rp][k][c]);
    }
    rp ^= 1;
}

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

// ---------------------------------------------------------------- geometry helpers
struct Cell {
    int c, i, j, W, E;
    bool south, north; // internal south / north faces
    bool xEfirst;      // east before west in face order (first column)
    bool yNfirst;      // north before south (bottom row of a multi-row mesh)
};

// row of a cell or y face index (idx / nx), without an integer division: exact while
// (idx + 0.5) / nx stays clear of an integer by more than the FP32 rounding, i.e. for
// any index below 2^21
__device__ __forceinline__ int rowOf(const DevClass &C, int idx) {
    return __float2int_rd((static_cast<float>(idx) + 0.5f) * __frcp_rn(static_cast<float>(C.nx)));
}
// the east neighbour of the cell owning x face f (periodic in x)
__device__ __forceinline__ int eastOf(const DevClass &C, int f) {
    return (f - rowOf(C, f) * C.nx == C.nx - 1) ? f - C.nx + 1 : f + 1;
}

__device__ __forceinline__ Cell cellOf(const DevClass &C, int c) {
    Cell q;
    q.c = c;
    q.j = rowOf(C, c);
    q.i = c - q.j * C.nx;
    q.W = q.i == 0 ? c + C.nx - 1 : c - 1;
    q.E = q.i == C.nx - 1 ? c - C.nx + 1 : c + 1;
    q.south = q.j > 0;
    q.north = q.j < C.ny - 1;
    q.xEfirst = q.i == 0;
    q.yNfirst = q.j == 0 && C.ny > 1;
    return q;
}

// accumulate onto a running value in face order
__device__ __forceinline__ double accum4(const Cell &q, double acc, double tW, double tE, double tS,
                                         double tN) {
    const double x1 = q.xEfirst ? tE : tW, x2 = q.xEfirst ? tW : tE;
    const double y1 = q.yNfirst ? tN : tS, y2 = q.yNfirst ? tS : tN;
    return (((acc + x1) + x2) + y1) + y2;
}

// column of wall values of a wall cell: bottom 0 .. nx - 1, top nx .. 2 nx - 1 (a cell
// touching both walls keeps the top one)
__device__ __forceinline__ int wallSlot(const DevClass &C, const Cell &q) {
    return q.i + (q.j == C.ny - 1 ? C.nx : 0);
}

// Geometry of a cell's Green-Gauss gradients (Field.hpp:178-212), shared by all fields:
// the interpolation weights (owner side) and outward area vectors of its faces, 1 / volume.
// At a wall face the weight picks the neighbour value, which grad() takes from the wall.
struct GradGeo {
    double wW, wE, wS, wN, xW, yW, xE, yE, xS, yS, xN, yN, iV;
    __device__ __forceinline__ GradGeo(const DevClass &C, const Cell &q) {
        const int c = q.c, fS = C.n + c, fN = fS + C.nx;
        wW = __ldg(C.fw + q.W);
        wE = __ldg(C.fw + c);
        wS = q.south ? __ldg(C.fw + fS) : 1.0;
        wN = q.north ? __ldg(C.fw + fN) : 0.0;
        xW = __ldg(C.fsx + q.W);
        yW = __ldg(C.fsy + q.W);
        xE = __ldg(C.fsx + c);
        yE = __ldg(C.fsy + c);
        xS = __ldg(C.fsx + fS);
        yS = __ldg(C.fsy + fS);
        if (q.south) { // owner below: outward is the other way
            xS = -xS;
            yS = -yS;
        }
        xN = __ldg(C.fsx + fN);
        yN = __ldg(C.fsy + fN);
        iV = __ldg(C.ivol + c);
    }
    // gradient from the cell's value and its neighbours' (S, N: the wall value at a wall).
    // The products of the x pair are rounded before they are added, so that they cancel
    // exactly where the flow does not vary along x.
    __device__ __forceinline__ void grad(double pc, double pW, double pE, double pS, double pN,
                                         double &gx, double &gy) const {
        const double fW = pW * wW + pc * (1.0 - wW), fE = pc * wE + pE * (1.0 - wE);
        const double fS = pS * wS + pc * (1.0 - wS), fN = pc * wN + pN * (1.0 - wN);
        const double tx = __dmul_rn(xE, fE) - __dmul_rn(xW, fW);
        const double ty = __dmul_rn(yE, fE) - __dmul_rn(yW, fW);
        gx = ((tx + __dmul_rn(xS, fS)) + __dmul_rn(xN, fN)) * iV;
        gy = ((ty + __dmul_rn(yS, fS)) + __dmul_rn(yN, fN)) * iV;
    }
    // the same of a field with wall values bS, bN
    __device__ __forceinline__ void of(const Cell &q, int nx, const double *phi, double bS, double bN,
                                       double &gx, double &gy) const {
        const int c = q.c;
        grad(phi[c], phi[q.W], phi[q.E], q.south ? phi[c - nx] : bS, q.north ? phi[c + nx] : bN, gx,
             gy);
    }
};

// Owner and neighbour cell of face f (x faces, then y faces); false for a wall face.
__device__ __forceinline__ bool faceCells(const DevClass &C, int f, int &o, int &q) {
    if (f < C.n) {
        o = f;
        q = eastOf(C, f);
        return true;
    }
    q = f - C.n;
    o = q - C.nx;
    return o >= 0 && q < C.n;
}

// Deferred correction F (phi_f - phi_up) of the limitedLinearUpwind face value (:495-552):
// phi_up + 0.5 psi(r) (phi_dn - phi_up) with r = 2 (grad phi)_up . d / (phi_dn - phi_up) - 1.
// dphi = phi_q - phi_o, d the vector from o to q: with q upwind both change sign in r.
__device__ __forceinline__ double limitedCorr(double F, double dphi, double gx, double gy, double dx,
                                              double dy) {
    if (!(fabs(dphi) > 1e-300) || F == 0.0)
        return 0.0;
    const double r = 2.0 * (gx * dx + gy * dy) / dphi - 1.0;
    const double psi = r > 0.0 ? (r * r + r) / (r * r + 1.0) : 0.0;
    return 0.5 * psi * (fabs(F) * dphi);
}

// matrix row times x in the reference's matvec order (diagonal first, then faces)
__device__ __forceinline__ double rowDot(const Cell &q, const double *d, const double *aW,
                                         const double *aE, const double *aS, const double *aN,
                                         const double *x, int nx) {
    const int c = q.c;
    const double tW = aW[c] * x[q.W], tE = aE[c] * x[q.E];
    const double tS = q.south ? aS[c] * x[c - nx] : 0.0;
    const double tN = q.north ? aN[c] * x[c + nx] : 0.0;
    return accum4(q, d[c] * x[c], tW, tE, tS, tN);
}

// The cells a thread owns in every per-cell sweep: c = thread, thread + threads, ...
// (a warp's loads of one sweep cover whole cache lines; contiguous blocks of cells per
// thread measured 12 % slower per outer iteration at 1536 cells). Every per-cell
// loop of a solve uses this one assignment, so a thread may read its own writes of
// an earlier loop without a barrier.
#define FOR_OWN(c, count) for (int c = gTid(), ts_ = gThreads(); c < (count); c += ts_)
#define FOR_CELLS(c) FOR_OWN(c, n)

// ---------------------------------------------------------------- inner linear solvers
// The Krylov and AMG routines are templated on the value type T of their
// vectors and matrices: T = double for the plain FP64 form, where they work
// directly on the arrays the assembly wrote; T = float for the mixed form,
// which solves for an FP32 correction inside an FP64 residual-refinement loop
// (mixedSolve below). Scalar coefficients and every reduction stay FP64.

// the five coefficient arrays of a 5-point system, held by value in registers
template <typename T> struct Mat {
    const T *d, *aW, *aE, *aS, *aN;
};
template <typename T> __device__ __forceinline__ Mat<T> matOf(const KW<T> &K) {
    return Mat<T>{K.d, K.aW, K.aE, K.aS, K.aN};
}

// row of a 5-point system times x, diagonal first then faces in the reference's
// matvec order (LinearSystem::matvec, LinearSolver.hpp:99-108)
template <typename T>
__device__ __forceinline__ T rowDotT(const Cell &q, const Mat<T> &M, const T *x, int nx) {
    const int c = q.c;
    const T tW = M.aW[c] * x[q.W], tE = M.aE[c] * x[q.E];
    const T tS = q.south ? M.aS[c] * x[c - nx] : T(0);
    const T tN = q.north ? M.aN[c] * x[c + nx] : T(0);
    const T x1 = q.xEfirst ? tE : tW, x2 = q.xEfirst ? tW : tE;
    const T y1 = q.yNfirst ? tN : tS, y2 = q.yNfirst ? tS : tN;
    return (((M.d[c] * x[c] + x1) + x2) + y1) + y2;
}

// Right-Jacobi BiCGSTAB (LinearSolver.hpp:251-345). K.r holds b - A x0 on entry and
// r0n its norm; x is updated in place.
template <typename T>
__device__ __noinline__ LinRes bicgstabT(Shared &S, int &rp, const KW<T> &K, T *x, double r0n,
                                         int maxIter, double tol) {
    const DevClass &C = S.C;
    const int n = C.n, nx = C.nx;
    LinRes res{0, 0.0, r0n, false};
    if (r0n < 1e-30) {
        res.converged = true;
        return res;
    }
    T *r = K.r, *rh = K.rh, *p = K.pv, *v = K.v, *s = K.s, *t = K.t, *ph = K.ph, *sh = K.sh,
      *rd = K.rd;
    const Mat<T> M = matOf(K);
    double acc[1];
    sumOver(acc, S, rp, n, [&](int c) {
        rh[c] = r[c];
        p[c] = T(0);
        v[c] = T(0);
        const T dc = M.d[c];
        rd[c] = (fabs(double(dc)) > 1e-30) ? T(1) / dc : T(1); // jacobiPrecond as a product
        acc[0] += double(r[c]) * double(r[c]);
    });
    double rhoN = acc[0], rho = 1, alpha = 1, omega = 1;
    for (int it = 0; it < maxIter; ++it) {
        if (fabs(rhoN) < 1e-30)
            break;
        const double beta = (rhoN / (rho + 1e-30)) * (alpha / (omega + 1e-30));
        FOR_CELLS(c) {
            const T pc = r[c] + T(beta) * (p[c] - T(omega) * v[c]);
            p[c] = pc;
            ph[c] = pc * rd[c];
        }
        SYNC();
        double a1[1];
        sumOver(a1, S, rp, n, [&](int c) {
            const Cell q = cellOf(C, c);
            const T vc = rowDotT(q, M, ph, nx);
            v[c] = vc;
            a1[0] += double(rh[c]) * double(vc);
        });
        const double rv = a1[0];
        if (fabs(rv) < 1e-30)
            break;
        alpha = rhoN / rv;
        double a2[1];
        sumOver(a2, S, rp, n, [&](int c) {
            const T sc = r[c] - T(alpha) * v[c];
            s[c] = sc;
            sh[c] = sc * rd[c];
            a2[0] += double(sc) * double(sc);
        });
        const double sn = sqrt(a2[0]);
        if (sn / r0n < tol) {
            FOR_CELLS(c) x[c] += T(alpha) * ph[c];
            SYNC();
            res.iterations = it + 1;
            res.finalRes = sn / r0n;
            res.converged = true;
            return res;
        }
        double a3[2];
        sumOver(a3, S, rp, n, [&](int c) {
            const Cell q = cellOf(C, c);
            const T tc = rowDotT(q, M, sh, nx);
            t[c] = tc;
            a3[0] += double(tc) * double(tc);
            a3[1] += double(tc) * double(s[c]);
        });
        const double tt = a3[0];
        omega = (tt > 1e-30) ? a3[1] / tt : 0.0;
        double a4[2];
        sumOver(a4, S, rp, n, [&](int c) {
            x[c] += T(alpha) * ph[c] + T(omega) * sh[c];
            const T rc = s[c] - T(omega) * t[c];
            r[c] = rc;
            a4[0] += double(rc) * double(rc);
            a4[1] += double(rh[c]) * double(rc);
        });
        const double rn = sqrt(a4[0]);
        res.iterations = it + 1;
        res.finalRes = rn / r0n;
        if (res.finalRes < tol) {
            res.converged = true;
            return res;
        }
        if (fabs(omega) < 1e-30)
            break;
        rho = rhoN;
        rhoN = a4[1];
    }
    SYNC();
    return res;
}

// ---------------------------------------------------------------- AMG V-cycle
template <typename T> __device__ __forceinline__ T level0EntryT(const KW<T> &K, int n, int e) {
    const int slot = e / n, c = e - slot * n;
    const T *a = slot == 0 ? K.d : slot == 1 ? K.aW : slot == 2 ? K.aE : slot == 3 ? K.aS : K.aN;
    return a[c];
}

// The levels of at most kLocalRows rows: every CTA of a cluster runs them whole, on vectors
// of its own in shared memory and with its own barrier (a cluster barrier costs about 520
// cycles, a CTA barrier 60). The threads that share a level, and a level's vectors (b, xa,
// xb, r, 1/diag).
__device__ __forceinline__ bool localLevel(const Shared &S, int l) {
    return kCluster && l >= S.C.locLevel;
}
__device__ __forceinline__ int levelTid(const Shared &S, int l) {
    return localLevel(S, l) ? threadIdx.x : gTid();
}
__device__ __forceinline__ int levelThreads(const Shared &S, int l) {
    return localLevel(S, l) ? blockDim.x : gThreads();
}
__device__ __forceinline__ void levelSync(const Shared &S, int l) {
    if (localLevel(S, l))
        __syncthreads();
    else
        SYNC();
}
template <typename T>
__device__ __forceinline__ T *levelVec(const Shared &S, const KW<T> &K, int l) {
    const int off = S.C.lev[l].vecOff;
    if (localLevel(S, l))
        return reinterpret_cast<T *>(S.locVec) + (off - S.C.lev[S.C.locLevel].vecOff);
    return K.amgVec + off;
}

// In-place inverse of the m x m matrix A (row-major, m <= kMaxCoarse; Gauss-Jordan, SPD: no
// pivoting) by the CTA's first 512 threads: each holds a tile of 8 x 4 entries, 16 rows and 32
// columns apart, and a pivot's row and column pass through shared memory (alternating
// buffers, one barrier per pivot). The inverse goes to out with leading dimension ld.
// Bound by issue and the barrier: a sweep over [A | I] in global memory moved 2 m^2 doubles in
// and out per pivot, 375 us for 96 rows.
constexpr int kInvThreads = 512;
__device__ __noinline__ void invertTiled(Shared &S, const double *A, int m, double *out, int ld) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double a[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = ty + 16 * i, c = tx + 32 * j;
            a[i][j] = r < m && c < m ? A[r * m + c] : 0.0;
        }
    // rows and columns of the pivot, alternating: 4 x kMaxCoarse doubles
    double *buf = S.coarse;
    auto publish = [&](int p) {
        double *row = buf + (p & 1) * 2 * kMaxCoarse, *col = row + kMaxCoarse;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (ty + 16 * i == p)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    row[tx + 32 * j] = a[i][j];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (tx + 32 * j == p)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    col[ty + 16 * i] = a[i][j];
        groupSync(kInvThreads);
    };
    publish(0);
    for (int p = 0; p < m; ++p) {
        const double *row = buf + (p & 1) * 2 * kMaxCoarse, *col = row + kMaxCoarse;
        const double inv = 1.0 / row[p];
        double pr[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            pr[j] = row[tx + 32 * j] * inv;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (16 * i >= m)
                break;
            const double f = col[ty + 16 * i];
            const bool own = ty + 16 * i == p;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double v = tx + 32 * j == p ? -f * inv : a[i][j] - f * pr[j];
                a[i][j] = own ? (tx + 32 * j == p ? inv : pr[j]) : v;
            }
        }
        if (p + 1 < m)
            publish(p + 1);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = ty + 16 * i, c = tx + 32 * j;
            if (r < m && c < m)
                out[r * ld + c] = a[i][j];
        }
}

// Galerkin values of every coarse level from the current pressure system, the
// reciprocal diagonals of the smoothed levels, then the inverse of the coarsest
// level (Gauss-Jordan, SPD: no pivoting): in place by one warp, one row per lane,
// when it has at most 32 rows; above that (up to 128) in register tiles (invertTiled), in
// CTAs of fewer than 512 threads by sweeps over [A | I] between two workspace buffers. (One warp
// with two rows per lane was measured 17 % slower per outer iteration at 1536
// cells: 128 dependent updates per lane and pivot against 16 per thread.) The
// inverse is FP64 in both forms.
template <typename T> __device__ __noinline__ void amgRefreshT(Shared &S, const KW<T> &K) {
    const DevClass &C = S.C;
    const Work &W = S.W;
    const int L = C.nlev;
    for (int l = 0; l + 1 < L; ++l) {
        const DevAmgLevel &F = C.lev[l];
        const DevAmgLevel &Q = C.lev[l + 1];
        T *cv = K.amgVal + Q.valOff;
        const T *fv = K.amgVal + F.valOff;
        // the first Galerkin sums cancel strongly (diagonal against off-diagonals of
        // one aggregate), so they are always formed from the FP64 finest matrix
        FOR_OWN(e, Q.nnz) {
            double s = 0.0;
            for (int k = __ldg(F.gPtr + e); k < __ldg(F.gPtr + e + 1); ++k) {
                const double v = (l == 0) ? level0EntryT(S.K64, C.n, __ldg(F.gSrc + k))
                                          : double(fv[__ldg(F.gSrc + k)]);
                s += __ldg(F.gW + k) * v;
            }
            cv[e] = T(s);
        }
        SYNC();
    }
    for (int l = 1; l + 1 < L; ++l) {
        const DevAmgLevel &Lv = C.lev[l];
        const T *val = K.amgVal + Lv.valOff;
        T *rdl = levelVec(S, K, l) + 4 * Lv.n;
        const int ts = levelThreads(S, l);
        for (int i = levelTid(S, l); i < Lv.n; i += ts)
            rdl[i] = T(1) / val[__ldg(Lv.diagPos + i)];
    }
    const DevAmgLevel &Q = C.lev[L - 1];
    const int m = Q.n; // at most kMaxCoarse = 128 rows (the set-up rejects more)
    const T *qv = K.amgVal + Q.valOff;
    if (m <= 32) {
        double *a = S.coarse;
        for (int e = threadIdx.x; e < m * m; e += blockDim.x)
            a[e] = 0.0;
        __syncthreads();
        if (L == 1) {
            for (int r = threadIdx.x; r < m; r += blockDim.x) {
                const Cell q = cellOf(C, r);
                a[r * m + r] += double(K.d[r]);
                a[r * m + q.W] += double(K.aW[r]);
                a[r * m + q.E] += double(K.aE[r]);
                if (q.south)
                    a[r * m + r - C.nx] += double(K.aS[r]);
                if (q.north)
                    a[r * m + r + C.nx] += double(K.aN[r]);
            }
        } else {
            for (int r = threadIdx.x; r < m; r += blockDim.x)
                for (int k = 0; k < Q.width; ++k) {
                    const int e = ellRow(r, Q.width) + 32 * k, c = __ldg(Q.ecol + e);
                    if (c >= 0)
                        a[r * m + c] = double(qv[e]);
                }
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const int r = threadIdx.x;
            for (int k = 0; k < m; ++k) {
                const double p = 1.0 / a[k * m + k];
                const double f = (r < m) ? a[r * m + k] : 0.0;
                __syncwarp();
                if (r < m && r != k) {
                    for (int j = 0; j < m; ++j)
                        if (j != k)
                            a[r * m + j] -= f * a[k * m + j] * p;
                    a[r * m + k] = -f * p;
                }
                __syncwarp();
                if (r == k) {
                    for (int j = 0; j < m; ++j)
                        if (j != k)
                            a[k * m + j] *= p;
                    a[k * m + k] = p;
                }
                __syncwarp();
            }
        }
        SYNC();
        return;
    }
    if (ctaRank() != 0) { // the inverse is the work of one CTA
        SYNC();
        return;
    }
    // m x 2m [A | I], row-major; the inverse ends in the right half of dense0 (the tiled
    // inversion takes A alone, in dense1)
    const bool tiled = static_cast<int>(blockDim.x) >= kInvThreads;
    const int m2 = tiled ? m : 2 * m;
    double *A0 = tiled ? W.dense1 : W.dense0, *A1 = W.dense1;
    for (int e = threadIdx.x; e < m * m2; e += blockDim.x)
        A0[e] = !tiled && ((e % m2) == m + e / m2) ? 1.0 : 0.0;
    __syncthreads();
    if (L == 1) {
        for (int r = threadIdx.x; r < m; r += blockDim.x) {
            const Cell q = cellOf(C, r);
            A0[r * m2 + r] += double(K.d[r]);
            A0[r * m2 + q.W] += double(K.aW[r]);
            A0[r * m2 + q.E] += double(K.aE[r]);
            if (q.south)
                A0[r * m2 + r - C.nx] += double(K.aS[r]);
            if (q.north)
                A0[r * m2 + r + C.nx] += double(K.aN[r]);
        }
    } else {
        for (int r = threadIdx.x; r < m; r += blockDim.x)
            for (int k = 0; k < Q.width; ++k) {
                const int e = ellRow(r, Q.width) + 32 * k, c = __ldg(Q.ecol + e);
                if (c >= 0)
                    A0[r * m2 + c] = double(qv[e]);
            }
    }
    __syncthreads();
    if (tiled) {
        if (threadIdx.x < kInvThreads)
            invertTiled(S, A0, m, W.dense0 + m, 2 * m);
        SYNC();
        return;
    }
    // the (row, column) of a thread's entries advance by the CTA width without a division
    const int dq = static_cast<int>(blockDim.x) / m2, dr = static_cast<int>(blockDim.x) - dq * m2;
    const int r0 = static_cast<int>(threadIdx.x) / m2, c0 = static_cast<int>(threadIdx.x) - r0 * m2;
    for (int piv = 0; piv < m; ++piv) {
        const double inv = 1.0 / A0[piv * m2 + piv];
        int r = r0, col = c0;
        for (int e = threadIdx.x; e < m * m2; e += blockDim.x) {
            const double pr = A0[piv * m2 + col] * inv;
            A1[e] = (r == piv) ? pr : A0[e] - A0[r * m2 + piv] * pr;
            r += dq;
            col += dr;
            if (col >= m2) {
                col -= m2;
                ++r;
            }
        }
        __syncthreads();
        double *tmp = A0;
        A0 = A1;
        A1 = tmp;
    }
    if (A0 != W.dense0) { // keep the inverse in dense0
        for (int e = threadIdx.x; e < m * m2; e += blockDim.x)
            W.dense0[e] = A0[e];
    }
    SYNC();
}

// Sum over the slots k = first, first + step, ... (< width) of one ELL row of
// coef(k) * vec(col(k)) for columns >= 0, k ascending. The loads of four slots are
// issued before their products are added (padding slots load entry 0 and add
// nothing), so a wide row costs a few load latencies, not one per slot.
template <typename T, typename C, typename V>
__device__ __forceinline__ T ellDot(const int32_t *cols, const C *coef, const V *vec, int width,
                                    int row, int first = 0, int step = 1) {
    cols += ellRow(row, width);
    coef += ellRow(row, width);
    T s = T(0);
    int k = first;
    for (; k + 3 * step < width; k += 4 * step) {
        int c[4];
        T v[4], x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            c[u] = __ldg(cols + (k + u * step) * 32);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            v[u] = T(coef[(k + u * step) * 32]);
            x[u] = T(vec[c[u] < 0 ? 0 : c[u]]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c[u] >= 0)
                s += v[u] * x[u];
    }
    if (k + step < width) {
        const int c0 = __ldg(cols + k * 32), c1 = __ldg(cols + (k + step) * 32);
        const T v0 = T(coef[k * 32]), v1 = T(coef[(k + step) * 32]);
        const T x0 = T(vec[c0 < 0 ? 0 : c0]), x1 = T(vec[c1 < 0 ? 0 : c1]);
        if (c0 >= 0)
            s += v0 * x0;
        if (c1 >= 0)
            s += v1 * x1;
        k += 2 * step;
    }
    if (k < width) {
        const int c = __ldg(cols + k * 32);
        if (c >= 0)
            s += T(coef[k * 32]) * T(vec[c]);
    }
    return s;
}

// Threads per row of a pass of nt threads over n rows: the largest power of two up to 32
// for which one pass still covers every row (1 when there are more rows than half the
// threads).
__device__ __forceinline__ int segOf(int n, int nt) {
    int seg = 1;
    while (seg < 32 && 2 * seg * n <= nt)
        seg *= 2;
    return seg;
}

// A pass over the rows of a small level with several threads per row (as many as one CTA could
// give each, so that the partial sums do not depend on the number of CTAs): lane j of a
// row's segment computes part(i, j, seg), the partial sum of the row's terms j,
// j + seg, ...; the partials are added by shuffles within the segment (a tree) and
// the segment's first lane calls use(i, total). Every one of the nt threads takes part, t
// its index (the shuffles need whole warps), so calls must be uniform across them. With one
// thread per row this is the plain row loop.
template <typename T, typename Part, typename Use>
__device__ __forceinline__ void segPass(int n, int t, int nt, Part part, Use use) {
    const int seg = segOf(n, blockDim.x), per = nt / seg;
    const int r = t / seg, j = t - r * seg;
    for (int base = 0; base < n; base += per) {
        const int i = base + r;
        T s = i < n ? part(i, j, seg) : T(0);
        for (int o = seg >> 1; o > 0; o >>= 1)
            s += __shfl_xor_sync(FULL, s, o);
        if (j == 0 && i < n)
            use(i, s);
    }
}

#include "rq_resident.cuh"

// z = M^-1 b at level 0 (b = K.r, z -> K.z): on every level above the coarsest,
// C.amgSweeps damped-Jacobi sweeps from zero, the residual, restriction by P^T (fused
// into the next level's first sweep), and after the coarse correction x + alpha P x_c
// (fused into the first post sweep) the same number of sweeps again (symmetric);
// a dense inverse on the coarsest level. Returns (r, z), reduced in the last phase.
// With one sweep a level costs three barrier-separated phases (two down, one up);
// with two, five. (Running the small coarse levels in one warp with warp barriers
// measured 15 % slower per outer iteration: one warp exposes the latency of its
// dependent loads that a CTA's many warps hide.)
template <typename T> __device__ __noinline__ double vcycleT(Shared &S, int &rp, const KW<T> &K) {
    const DevClass &C = S.C;
    const Work &W = S.W;
    const int L = C.nlev, n0 = C.n, nx = C.nx;
    const bool two = C.amgSweeps >= 2;
    const T om = T(C.amgW), al = T(C.amgAlpha);
    const Mat<T> M = matOf(K);
    T *const Krd = K.rd, *const Kr = K.r, *const Kz = K.z, *const Kxa = K.xa, *const Kxb = K.xb,
             *const Krr = K.rr, *const amgVal = K.amgVal;
    auto vb = [&](int l) { return levelVec(S, K, l); }; // b, xa, xb, r, 1/diag
    auto sync = [&](int l) { levelSync(S, l); };
    // residual of level l-1 restricted to row I of level l: sum_k R_Ik r_k (lane j of
    // the row's segment: the terms j, j + seg, ...)
    auto restrictPart = [&](int l, int I, int j, int seg) {
        const DevAmgLevel &F = C.lev[l - 1];
        const T *fr = (l == 1) ? Krr : vb(l - 1) + 3 * F.n;
        return ellDot<T>(F.rcol, F.rval, fr, F.rw, I, j, seg);
    };
    // the prolongated coarse correction at row i of level l: sum_k P_ik x_c
    auto prolong = [&](int l, int i) {
        const DevAmgLevel &Lv = C.lev[l];
        const T *xc = vb(l + 1) + 2 * C.lev[l + 1].n;
        return ellDot<T>(Lv.pcol, Lv.pval, xc, Lv.pw, i);
    };
    // one level of the down sweep; the pre-smoothed iterate ends in xa (one sweep) or
    // xb (two sweeps), the residual in rr. Coarse levels run several threads per row.
    auto down = [&](int l) {
        const DevAmgLevel &Lv = C.lev[l];
        const int n = Lv.n, t0 = levelTid(S, l), ts = levelThreads(S, l);
        if (l == 0) {
            FOR_OWN(i, n)
                Kxa[i] = om * Kr[i] * Krd[i];
            sync(l);
            const T *xs = Kxa;
            if (two) {
                FOR_OWN(i, n) {
                    const T ax = rowDotT(cellOf(C, i), M, Kxa, nx);
                    Kxb[i] = Kxa[i] + om * (Kr[i] - ax) * Krd[i];
                }
                sync(l);
                xs = Kxb;
            }
            FOR_OWN(i, n)
                Krr[i] = Kr[i] - rowDotT(cellOf(C, i), M, xs, nx);
            sync(l);
            return;
        }
        T *b = vb(l), *xa = b + n, *xb = b + 2 * n, *rr = b + 3 * n;
        const T *rd = b + 4 * n;
        const T *val = amgVal + Lv.valOff;
        segPass<T>(n, t0, ts, [&](int i, int j, int seg) { return restrictPart(l, i, j, seg); },
                   [&](int i, T bi) {
                       b[i] = bi;
                       xa[i] = om * bi * rd[i];
                   });
        sync(l);
        const T *xs = xa;
        if (two) {
            segPass<T>(n, t0, ts,
                       [&](int i, int j, int seg) {
                           return ellDot<T>(Lv.ecol, val, xa, Lv.width, i, j, seg);
                       },
                       [&](int i, T ax) { xb[i] = xa[i] + om * (b[i] - ax) * rd[i]; });
            sync(l);
            xs = xb;
        }
        segPass<T>(n, t0, ts,
                   [&](int i, int j, int seg) {
                       return ellDot<T>(Lv.ecol, val, xs, Lv.width, i, j, seg);
                   },
                   [&](int i, T ax) { rr[i] = b[i] - ax; });
        sync(l);
    };
    // the coarsest level: restriction of the level above, then the dense inverse
    auto coarsest = [&]() {
        const int l = L - 1, t0 = levelTid(S, l), ts = levelThreads(S, l);
        const int m = C.lev[l].n, m2 = 2 * m;
        T *b = vb(l), *xb = b + 2 * m;
        if (L == 1) {
            FOR_OWN(i, m)
                b[i] = Kr[i];
        } else {
            segPass<T>(m, t0, ts, [&](int i, int j, int seg) { return restrictPart(l, i, j, seg); },
                       [&](int i, T bi) { b[i] = bi; });
        }
        sync(l);
        // the coarsest solve stays FP64 in both forms: the coarsest level of the
        // pinned all-Neumann pressure system is nearly singular, and an FP32
        // copy of its inverse loses the coarse correction
        const double *inv = (m <= 32) ? S.coarse : W.dense0 + m;
        const int ld = (m <= 32) ? m : m2;
        segPass<double>(m, t0, ts,
                        [&](int i, int j, int seg) {
                            const double *row = inv + i * ld;
                            double s = 0.0;
                            for (int k = j; k < m; k += seg)
                                s += row[k] * double(b[k]);
                            return s;
                        },
                        [&](int i, double s) { xb[i] = T(s); });
        sync(l);
    };
    // one level of the up sweep (levels >= 1; level 0 ends in the reduction below):
    // x = x_pre + alpha P x_c, then the post sweeps; the result ends in xb. With a
    // piecewise-constant P (one coarse row per fine row) x is formed inside the first
    // sweep; with a smoothed P it is formed in a phase of its own, in place of x_pre (not
    // in the residual's slot: see upRes), so that the sweep over a wide coarse row loads
    // each neighbour's x once instead of re-forming it from P.
    auto up = [&](int l) {
        const DevAmgLevel &Lv = C.lev[l];
        const int n = Lv.n, t0 = levelTid(S, l), ts = levelThreads(S, l);
        T *b = vb(l), *xa = b + n, *xb = b + 2 * n;
        const T *rd = b + 4 * n;
        T *xpre = two ? xb : xa;
        T *out = two ? xa : xb;
        const T *val = amgVal + Lv.valOff;
        if (Lv.pw > 1) {
            for (int i = t0; i < n; i += ts)
                xpre[i] += al * prolong(l, i);
            sync(l);
            segPass<T>(n, t0, ts,
                       [&](int i, int j, int seg) {
                           return ellDot<T>(Lv.ecol, val, xpre, Lv.width, i, j, seg);
                       },
                       [&](int i, T ax) { out[i] = xpre[i] + om * (b[i] - ax) * rd[i]; });
        } else {
            for (int i = t0; i < n; i += ts) {
                const T x0 = xpre[i] + al * prolong(l, i);
                T ax = T(0);
                for (int k = 0; k < Lv.width; ++k) {
                    const int e = ellRow(i, Lv.width) + 32 * k, jj = __ldg(Lv.ecol + e);
                    if (jj >= 0)
                        ax += val[e] * (xpre[jj] + al * prolong(l, jj));
                }
                out[i] = x0 + om * (b[i] - ax) * rd[i];
            }
        }
        sync(l);
        if (two) {
            segPass<T>(n, t0, ts,
                       [&](int i, int j, int seg) {
                           return ellDot<T>(Lv.ecol, val, xa, Lv.width, i, j, seg);
                       },
                       [&](int i, T ax) { xb[i] = xa[i] + om * (b[i] - ax) * rd[i]; });
            sync(l);
        }
    };
    bool lean = false;
    if constexpr (std::is_same_v<T, double>)
        lean = S.lean;
    if (L > 1)
        down(0);
    if (lean) {
        if constexpr (std::is_same_v<T, double>)
            coarseRes<false>(S, L > 1 ? Krr : Kr);
    } else {
        for (int l = 1; l + 1 < L; ++l)
            down(l);
        coarsest();
        for (int l = L - 2; l >= 1; --l)
            up(l);
    }
    double rz = 0.0;
    if (L > 1 && (lean || C.lev[0].pw > 1)) { // level 0, smoothed P: x = x_pre + alpha P x_c in a
        // sweep of its own (in place of x_pre: see upRes), then the
        // post sweep(s) read it (each x once, not re-formed at every neighbour)
        const int n = C.lev[0].n;
        T *x = two ? Kxb : Kxa;
        if (lean) {
            if constexpr (std::is_same_v<T, double>) {
                const ResLevel &R = S.RL[0];
                const double *xc = S.RL[1].x;
                FOR_OWN(i, n)
                    x[i] += al * rowRes(R.pc, R.pv, xc, R.pw, i);
            }
        } else {
            FOR_OWN(i, n)
                x[i] += al * prolong(0, i);
        }
        SYNC();
        auto sweep = [&](const T *from, T *to, int i) { // a damped-Jacobi sweep's row
            const T ax = rowDotT(cellOf(C, i), M, from, nx);
            const T zi = from[i] + om * (Kr[i] - ax) * Krd[i];
            to[i] = zi;
            return zi;
        };
        double a[1];
        if (two) {
            FOR_OWN(i, n)
                sweep(x, Kxa, i);
            SYNC();
            sumOver(a, S, rp, n, [&](int i) { a[0] += double(Kr[i]) * double(sweep(Kxa, Kz, i)); });
        } else {
            sumOver(a, S, rp, n, [&](int i) { a[0] += double(Kr[i]) * double(sweep(x, Kz, i)); });
        }
        rz = a[0];
    } else if (L > 1) { // level 0, piecewise-constant P: prolongation fused into the
        // first post sweep (then the second)
        const int n = C.lev[0].n;
        const T *xprev = two ? Kxb : Kxa;
        auto first = [&](T *to, int i) {
            const T xi = xprev[i] + al * prolong(0, i);
            const Cell q = cellOf(C, i);
            const int c = i;
            auto X = [&](int jj) { return xprev[jj] + al * prolong(0, jj); };
            const T tW = M.aW[c] * X(q.W), tE = M.aE[c] * X(q.E);
            const T tS = q.south ? M.aS[c] * X(c - nx) : T(0);
            const T tN = q.north ? M.aN[c] * X(c + nx) : T(0);
            const T x1 = q.xEfirst ? tE : tW, x2 = q.xEfirst ? tW : tE;
            const T y1 = q.yNfirst ? tN : tS, y2 = q.yNfirst ? tS : tN;
            const T ax = (((M.d[c] * xi + x1) + x2) + y1) + y2;
            const T zi = xi + om * (Kr[i] - ax) * Krd[c];
            to[i] = zi;
            return zi;
        };
        double a[1];
        if (two) {
            FOR_OWN(i, n)
                first(Kxa, i);
            SYNC();
            sumOver(a, S, rp, n, [&](int i) {
                const T ax = rowDotT(cellOf(C, i), M, Kxa, nx);
                const T zi = Kxa[i] + om * (Kr[i] - ax) * Krd[i];
                Kz[i] = zi;
                a[0] += double(Kr[i]) * double(zi);
            });
        } else {
            sumOver(a, S, rp, n, [&](int i) { a[0] += double(Kr[i]) * double(first(Kz, i)); });
        }
        rz = a[0];
    } else {
        const T *xb = vb(0) + 2 * C.lev[0].n;
        double a[1];
        sumOver(a, S, rp, n0, [&](int i) {
            Kz[i] = xb[i];
            a[0] += double(Kr[i]) * double(xb[i]);
        });
        rz = a[0];
    }
    return rz;
}

// The sweeps of one PCG iteration as functions of their own, so that the PCG loop
// itself keeps only a few scalars live across the V-cycle call (every value live
// across a call is saved to and reloaded from local memory around it).
// Ap = A p; returns (p, Ap).
template <typename T> __device__ __noinline__ double pcgMatvec(Shared &S, int &rp, const KW<T> &K) {
    const DevClass &C = S.C;
    const int n = C.n, nx = C.nx;
    const Mat<T> M = matOf(K);
    const T *p = K.pv;
    T *Ap = K.v;
    double a[1];
    sumOver(a, S, rp, n, [&](int c) {
        const T v = rowDotT(cellOf(C, c), M, p, nx);
        Ap[c] = v;
        a[0] += double(p[c]) * double(v);
    });
    return a[0];
}
// x += alpha p, r -= alpha Ap; returns (r, r)
template <typename T>
__device__ __noinline__ double pcgUpdate(Shared &S, int &rp, const KW<T> &K, T *x, double alpha) {
    const int n = S.C.n;
    const T *p = K.pv, *Ap = K.v;
    T *r = K.r;
    double a[1];
    sumOver(a, S, rp, n, [&](int c) {
        x[c] += T(alpha) * p[c];
        const T rc = r[c] - T(alpha) * Ap[c];
        r[c] = rc;
        a[0] += double(rc) * double(rc);
    });
    return a[0];
}
// z = r / diag; returns (r, z)
template <typename T> __device__ __noinline__ double pcgJacobi(Shared &S, int &rp, const KW<T> &K) {
    const int n = S.C.n;
    const T *r = K.r, *rdv = K.rd;
    T *z = K.z;
    double a[1];
    sumOver(a, S, rp, n, [&](int c) {
        z[c] = r[c] * rdv[c];
        a[0] += double(r[c]) * double(z[c]);
    });
    return a[0];
}
// p = z + beta p (beta 0: p = z), then a barrier
template <typename T> __device__ __noinline__ void pcgDirection(Shared &S, const KW<T> &K, double beta) {
    const int n = S.C.n;
    const T *z = K.z;
    T *p = K.pv;
    if (beta == 0.0) {
        FOR_CELLS(c) p[c] = z[c];
    } else {
        FOR_CELLS(c) p[c] = z[c] + T(beta) * p[c];
    }
    SYNC();
}
// x += alpha p, r -= alpha Ap; returns (r, r) and the sum of r (the mixed form's
// deflation of the constant vector needs it)
struct Two {
    double a, b;
};
template <typename T>
__device__ __noinline__ Two pcgUpdateSum(Shared &S, int &rp, const KW<T> &K, T *x, double alpha) {
    const int n = S.C.n;
    const T *p = K.pv, *Ap = K.v;
    T *r = K.r;
    double a[2];
    sumOver(a, S, rp, n, [&](int c) {
        x[c] += T(alpha) * p[c];
        const T rc = r[c] - T(alpha) * Ap[c];
        r[c] = rc;
        a[0] += double(rc) * double(rc);
        a[1] += double(rc);
    });
    return Two{a[0], a[1]};
}
// the sum of r (the first residual of a solve)
template <typename T> __device__ __noinline__ double sumOf(Shared &S, int &rp, const T *r) {
    const int n = S.C.n;
    double a[1];
    sumOver(a, S, rp, n, [&](int c) { a[0] += double(r[c]); });
    return a[0];
}

// z = M^-1 r of the mixed form: the FP32 V-cycle of S.K32 with the constant vector 1
// deflated in FP64. The pressure system is all-Neumann but for the pin of cell 0, so
// A 1 = rowsum0 e_0 and 1 spans its near-null space; FP32 coarse values round each
// coarse row sum (zero in exact arithmetic) by about 1e-7 of its diagonal, which is
// comparable to that mode's eigenvalue and spoils its coarse correction. So the
// constant mode is solved exactly in FP64 and the V-cycle sees only the rest
// (balancing: M^-1 = Q + (I - Q A) V (I - A Q), Q = 1 (1' A 1)^-1 1', SPD when V is):
//   r~ = r - (1'r) e_0,  y = V r~,  z = y + ((1'r) / rowsum0 - y_0) 1.
// sumR = 1'r; returns (r, z) and (r, z_previous) in FP64 (the latter for the flexible
// direction update: an FP32 V-cycle is symmetric only to its rounding).
template <typename T>
__device__ __noinline__ Two pcgPrecondF32(Shared &S, int &rp, const KW<T> &K, double sumR,
                                          double rowsum0) {
    const int n = S.C.n;
    {
        const KW<float> &F = S.K32;
        const T *r = K.r;
        FOR_CELLS(c) F.r[c] = float(c == 0 ? double(r[c]) - sumR : double(r[c]));
    }
    vcycleT<float>(S, rp, S.K32); // ends with a block reduction: F.z is complete
    const KW<float> &F = S.K32;
    const double shift = sumR / rowsum0 - double(F.z[0]);
    const T *r = K.r;
    T *z = K.z;
    double a[2];
    sumOver(a, S, rp, n, [&](int c) {
        const T zc = T(double(F.z[c]) + shift);
        a[1] += double(r[c]) * double(z[c]);
        z[c] = zc;
        a[0] += double(r[c]) * double(zc);
    });
    return Two{a[0], a[1]};
}

// PCG (LinearSolver.hpp:184-246 / :908-982) from x = 0 with the Jacobi or the AMG
// preconditioner; K.r holds b and r0n its norm, x receives the solution.
// With F32Precond the AMG V-cycle runs on the FP32 copies (S.K32) while PCG itself
// stays in T = double: the mixed form of the pressure solve.
template <typename T, bool F32Precond>
__device__ __noinline__ LinRes pcgT(Shared &S, int &rp, const KW<T> &K, T *x, double r0n,
                                    int maxIter, double tol, bool amg, bool refresh) {
    LinRes res{0, 0.0, r0n, false};
    if (r0n < 1e-30) {
        res.converged = true;
        return res;
    }
    {
        const int n = S.C.n;
        const T *d = K.d;
        T *rdv = K.rd;
        FOR_CELLS(c) {
            const T dc = d[c];
            rdv[c] = (fabs(double(dc)) > 1e-30) ? T(1) / dc : T(1);
            x[c] = T(0);
        }
        if constexpr (F32Precond) {
            if (amg) { // FP32 copy of the finest level for the FP32 V-cycle
                const KW<float> &F = S.K32;
                const Mat<T> M = matOf(K);
                FOR_CELLS(c) {
                    F.d[c] = float(M.d[c]);
                    F.aW[c] = float(M.aW[c]);
                    F.aE[c] = float(M.aE[c]);
                    F.aS[c] = float(M.aS[c]);
                    F.aN[c] = float(M.aN[c]);
                    F.rd[c] = (fabs(double(F.d[c])) > 1e-30) ? 1.0f / F.d[c] : 1.0f;
                }
                SYNC();
            }
        }
    }
    if (amg && refresh) {
        mark(S, 4);
        if constexpr (F32Precond)
            amgRefreshT<float>(S, S.K32);
        else {
            amgRefreshT(S, K); // begins with a barrier-separated phase
            if (S.lean)
                denseOrder(S);
        }
        mark(S, 5);
    } else {
        SYNC();
    }
    // the mixed form deflates the constant vector (pcgPrecondF32): the row sum of the
    // pinned row and the running sum of r
    double rowsum0 = 0.0, sumR = 0.0;
    if constexpr (F32Precond) {
        if (amg) {
            rowsum0 = double(K.d[0]) + double(K.aW[0]) + double(K.aE[0]) + double(K.aS[0]) +
                      double(K.aN[0]);
            sumR = sumOf(S, rp, K.r);
        }
    }
    // (r, z) of the new preconditioned residual; rzPrev receives (r, z_previous) where
    // the flexible update applies (the FP32 V-cycle), else 0
    double rzPrev = 0.0;
    auto precond = [&]() {
        if (!amg)
            return pcgJacobi(S, rp, K);
        if constexpr (F32Precond) {
            const Two u = pcgPrecondF32(S, rp, K, sumR, rowsum0);
            rzPrev = u.b;
            return u.a;
        } else {
            return vcycleT(S, rp, K);
        }
    };
    if constexpr (F32Precond) { // z_previous of the first direction: zero
        const int n = S.C.n;
        FOR_CELLS(c) K.z[c] = T(0);
    }
    double rz = precond();
    pcgDirection(S, K, 0.0);
    for (int it = 0; it < maxIter; ++it) {
        const double pAp = pcgMatvec(S, rp, K);
        if (fabs(pAp) < 1e-30) {
            res.breakdown = true;
            break;
        }
        double rr2;
        if constexpr (F32Precond) {
            const Two u = pcgUpdateSum(S, rp, K, x, rz / pAp);
            rr2 = u.a;
            sumR = u.b;
        } else {
            rr2 = pcgUpdate(S, rp, K, x, rz / pAp);
        }
        const double rn = sqrt(rr2);
        res.iterations = it + 1;
        res.finalRes = rn / r0n;
        if (res.finalRes < tol) {
            res.converged = true;
            return res;
        }
        const double rzNew = precond();
        // Fletcher-Reeves as the reference; Polak-Ribiere (flexible CG) around the
        // FP32 V-cycle
        pcgDirection(S, K, (rzNew - rzPrev) / (rz + 1e-30));
        rz = rzNew;
    }
    return res;
}

// Mixed form of one linear solve: FP32 Krylov (and AMG) iterations for a
// correction of the FP64 solution, with the residual of the FP64 system
// recomputed after each correction (iterative refinement) until it has dropped
// by tol relative to the initial residual or the iteration budget is spent.
// On entry W.b and W.r hold the FP64 right-hand side and b - A x (x = x64) and
// r0n its norm; initialRes is that FP64 norm, as in the plain form.
__device__ __noinline__ LinRes mixedSolve(Shared &S, int &rp, double *x64, double r0n, int maxIter,
                                          double tol, int kind, bool refresh) {
    const DevClass &C = S.C;
    const Work &W = S.W;
    const KW<float> &K = S.K32;
    const int n = C.n, nx = C.nx;
    LinRes out{0, 0.0, r0n, false};
    if (r0n < 1e-30) {
        out.converged = true;
        return out;
    }
    FOR_CELLS(c) {
        K.d[c] = float(W.d[c]);
        K.aW[c] = float(W.aW[c]);
        K.aE[c] = float(W.aE[c]);
        K.aS[c] = float(W.aS[c]);
        K.aN[c] = float(W.aN[c]);
        K.r[c] = float(W.r[c]);
    }
    SYNC();
    double rn = r0n;
    bool refreshNow = refresh;
    for (int round = 0; round < 8 && out.iterations < maxIter; ++round) {
        // the FP32 solve targets the remaining reduction of the FP64 residual
        const double innerTol = tol * r0n / rn;
        double an[1];
        sumOver(an, S, rp, n, [&](int c) { an[0] += double(K.r[c]) * double(K.r[c]); });
        const double r32n = sqrt(an[0]);
        LinRes in;
        FOR_CELLS(c) K.x[c] = 0.0f;
        SYNC();
        in = bicgstabT<float>(S, rp, K, K.x, r32n, maxIter - out.iterations, innerTol);
        (void)refreshNow;
        out.iterations += in.iterations;
        FOR_CELLS(c) x64[c] += double(K.x[c]);
        SYNC();
        double a[1];
        sumOver(a, S, rp, n, [&](int c) {
            const Cell q = cellOf(C, c);
            const double rc = W.b[c] - rowDot(q, W.d, W.aW, W.aE, W.aS, W.aN, x64, nx);
            W.r[c] = rc;
            K.r[c] = float(rc);
            a[0] += rc * rc;
        });
        rn = sqrt(a[0]);
        if (rn / r0n < tol) {
            out.converged = true;
            break;
        }
        if (in.iterations == 0 || !isfinite(rn))
            break;
    }
    out.finalRes = rn / r0n;
    return out;
}

// Linear-solve dispatch: the resident form where carve() set it up, else by the
// precision of the class. The result is complete in `out` (shared memory) after the
// caller's next barrier.
__device__ __forceinline__ void solveBicg(Shared &S, int &rp, double *x, double r0n, int maxIter,
                                          double tol, LinRes *out) {
    if (S.resWarps) {
        if (static_cast<int>(threadIdx.x) < 32 * S.resWarps)
            bicgstabRes(x, r0n, maxIter, tol, out);
        return;
    }
    *out = S.C.st.precision == kMixed
               ? mixedSolve(S, rp, x, r0n, maxIter, tol, kPBicgstab, false)
               : bicgstabT<double>(S, rp, S.K64, x, r0n, maxIter, tol);
}

// The AMG coarse values (Galerkin products and the coarsest inverse) are refreshed
// when the previous pressure solve degraded: more than 1.5x (+2) the PCG iterations
// of the solve right after the last refresh, or stopped short of its tolerance
// other than on the |p.Ap| < 1e-30 guard. That is the rule AMGSolver applies to its
// aggregation (LinearSolver.hpp:924-941), except that a guard exit does not count:
// late in a solve the p' right-hand side is round-off (|b| ~ 1e-15), PCG stops on the
// guard whatever the preconditioner, and fresh coarse values would not change that.
// The stale coarse operator stays SPD, so PCG remains valid; the finest level
// always uses the current matrix.
__device__ __forceinline__ LinRes solvePressure(Shared &S, int &rp, double *x, double r0n,
                                                int maxIter, double tol, int kind,
                                                int &needRefresh, int &itersAfterRefresh) {
    const bool amg = kind == kPAmg;
    const bool refresh = amg && needRefresh;
    LinRes res;
    const bool mixed = S.C.st.precision == kMixed;
    if (S.resWarps && (!amg || S.resAmg)) { // the resident forms
        if (refresh && r0n >= 1e-30) {
            mark(S, 4);
            amgRefreshT(S, S.K64);
            denseOrder(S);
            mark(S, 5);
        }
        if (amg)
            pcgRes<true>(x, r0n, maxIter, tol, &S.L.resP);
        else if (kind == kPPcg)
            pcgRes<false>(x, r0n, maxIter, tol, &S.L.resP);
        else if (static_cast<int>(threadIdx.x) < 32 * S.resWarps)
            bicgstabRes(x, r0n, maxIter, tol, &S.L.resP);
        SYNC();
        res = S.L.resP;
    } else if (kind == kPBicgstab)
        res = mixed ? mixedSolve(S, rp, x, r0n, maxIter, tol, kind, refresh)
                    : bicgstabT<double>(S, rp, S.K64, x, r0n, maxIter, tol);
    else if (mixed) // FP64 PCG, FP32 AMG V-cycle
        res = pcgT<double, true>(S, rp, S.K64, x, r0n, maxIter, tol, amg, refresh);
    else
        res = pcgT<double, false>(S, rp, S.K64, x, r0n, maxIter, tol, amg, refresh);
    if (amg && r0n >= 1e-30) {
        if (refresh) {
            needRefresh = 0;
            itersAfterRefresh = res.iterations;
        } else if (itersAfterRefresh <= 0) {
            itersAfterRefresh = res.iterations;
        } else if ((!res.converged && !res.breakdown) ||
                   res.iterations > 1.5 * itersAfterRefresh + 2) {
            needRefresh = 1;
        }
    }
    return res;
}

// ---------------------------------------------------------------- contraction estimate
// ContractionEstimate (SIMPLESolver.cpp:32-74) over a shared ring of samples;
// every warp evaluates the window maxima with shuffles (max is exact).
struct Est {
    double rate, remaining;
};
__device__ __forceinline__ Est estimate(const Shared &S, int e, int window, double negligible) {
    const int m = window < 2 ? 2 : window;
    const int cnt = S.cnt[e];
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    if (cnt < 2 * m)
        return {__longlong_as_double(0x7ff8000000000000LL), inf};
    const int lane = threadIdx.x & 31;
    double dNew = 0.0, dOld = 0.0;
    for (int l = lane; l < m; l += 32) {
        dNew = dmax(dNew, S.ring[e][(cnt - m + l) % kWindowCap]);
        dOld = dmax(dOld, S.ring[e][(cnt - 2 * m + l) % kWindowCap]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        dNew = dmax(dNew, __shfl_xor_sync(FULL, dNew, o));
        dOld = dmax(dOld, __shfl_xor_sync(FULL, dOld, o));
    }
    double rate;
    if (dOld <= 0.0)
        rate = dNew > 0.0 ? inf : 0.0;
    else
        rate = pow(dNew / dOld, 1.0 / m);
    double remaining;
    if (dNew <= negligible)
        remaining = dNew;
    else if (!(rate < 1.0))
        remaining = inf;
    else
        remaining = dNew * rate / (1.0 - rate);
    return {rate, remaining};
}

__device__ __forceinline__ void pushSample(Shared &S, int e, double v) {
    SYNC(); // everyone finished reading the ring
    if (threadIdx.x == 0) {
        S.ring[e][S.cnt[e] % kWindowCap] = v;
        S.cnt[e] += 1;
    }
    SYNC();
}

// ---------------------------------------------------------------- the solve
// Workspace placement: arrays in priority order go to the shared-memory arena
// while it has room (the hot Krylov/AMG vectors and the matrix first), the rest
// to this CTA's global workspace, which has a slot for every array.
__device__ void carve(Shared &S, double *ws, double *arena, long arenaDoubles) {
    const DevClass &C = S.C;
    const long n = C.n, nf = C.n + C.nfy;
    Work &W = S.W;
    double *g = ws;
    long used = 0;
    // the resident solvers where a thread can hold its cells in registers
    S.resWarps = 0;
    S.locVec = arena;
    const long arenaAll = arenaDoubles;
    if constexpr (kCluster) // the CTAs share every array; the arena holds the local levels
        arenaDoubles = 0;
    if (!kCluster && C.st.precision == kFP64 && static_cast<int>(blockDim.x) <= kResMaxThreads &&
        n <= static_cast<long>(kResCells) * blockDim.x && resExchange(n) <= arenaDoubles) {
        used = resExchange(n); // the exchange vectors start the arena
        S.resWarps = resThreads(n) / 32;
    }
    // and their V-cycle, whose level vectors come next
    const long vecs = (C.amgVecs + 31) / 32 * 32;
    S.resAmg = S.resWarps && C.resAmg && used + vecs <= arenaDoubles;
    S.lean = C.resAmg && C.st.precision == kFP64 && C.st.pSolver == kPAmg;
    auto take = [&](long cnt) {
        const long sz = (cnt + 31) / 32 * 32;
        double *gp = g;
        g += sz;
        if (used + sz <= arenaDoubles) {
            double *sp = arena + used;
            used += sz;
            return sp;
        }
        return gp;
    };
    double *resVec = arena + used;
    if (S.resAmg)
        used += vecs;
    // the general solvers' vectors: never touched where the resident forms cover all solves
    const bool covered = S.resWarps && (S.resAmg || C.st.pSolver != kPAmg);
    auto cold = [&](long cnt) {
        if (!covered)
            return take(cnt);
        double *gp = g;
        g += (cnt + 31) / 32 * 32;
        return gp;
    };
    auto takeF = [&](long cnt) { return reinterpret_cast<float *>(take((cnt + 1) / 2)); };
    const int m = C.lev[C.nlev - 1].n;
    const bool mixed = C.st.precision == kMixed;
    KW<float> &F = S.K32;
    if (mixed) { // the FP32 inner-solver storage is the hot set of the mixed form
        F.d = takeF(n);
        F.aW = takeF(n);
        F.aE = takeF(n);
        F.aS = takeF(n);
        F.aN = takeF(n);
        F.rd = takeF(n);
        F.r = takeF(n);
        F.pv = takeF(n);
        F.v = takeF(n);
        F.ph = takeF(n);
        F.s = takeF(n);
        F.sh = takeF(n);
        F.t = takeF(n);
        F.rh = takeF(n);
        F.x = takeF(n);
        F.amgVec = takeF(C.amgVecs);
        F.amgVal = takeF(C.amgVals);
        F.z = F.s;
        F.xa = F.t;
        F.xb = F.sh;
        F.rr = F.rh;
    }
    // tier 1: matrix and Krylov vectors
    W.d = take(n);
    W.aW = take(n);
    W.aE = take(n);
    W.aS = take(n);
    W.aN = take(n);
    W.r = take(n);
    if (mixed) { // the mixed form keeps only the FP64 vectors of the pressure PCG
        W.pv = take(n);
        W.v = take(n);
        W.z = take(n);
        W.rd = take(n);
    } else {
        W.pv = cold(n);
        W.v = cold(n);
        W.ph = cold(n);
        W.s = cold(n);
        W.sh = cold(n);
        W.t = cold(n);
        W.rh = cold(n);
        W.rd = cold(n);
        // the pressure PCG / V-cycle vectors share storage with the BiCGSTAB-only
        // vectors: the two solvers never run at the same time
        W.z = W.s;
        W.xa = W.t;
        W.xb = W.sh;
        W.rr = W.rh;
        // tier 2: AMG (vectors first: touched more often)
        W.amgVec = S.resAmg ? resVec : take(C.amgVecs);
        W.amgVal = take(C.amgVals);
        if (S.lean)
            resPlace(S, [&](long cnt) {
                const long sz = (cnt + 31) / 32 * 32;
                if (kCluster && used == 0)
                    used = C.locDoubles;
                if (used + sz > arenaAll)
                    return static_cast<double *>(nullptr);
                double *sp = arena + used;
                used += sz;
                return sp;
            });
    }
    // tier 3: solved fields and assembly inputs
    W.pp = take(n);
    W.Ux = take(n);
    W.Uy = take(n);
    W.k = take(n);
    W.w = take(n);
    W.b = take(n);
    W.aP = take(n);
    W.nuT = take(n);
    W.F1 = take(n);
    W.phi = take(nf);
    W.phiPred = take(nf);
    W.pCoeff = take(nf);
    W.fScr = take(nf);
    W.gPx = take(n);
    W.gPy = take(n);
    W.gUxx = take(n);
    W.gUxy = take(n);
    W.gUyx = take(n);
    W.gUyy = take(n);
    W.gKx = take(n);
    W.gKy = take(n);
    W.gWx = take(n);
    W.gWy = take(n);
    // tier 4
    W.p = take(n);
    W.F2 = take(n);
    W.Pk = take(n);
    W.CD = take(n);
    W.S = take(n);
    W.Uxp = take(n);
    W.Uyp = take(n);
    W.kOld = take(n);
    W.wOld = take(n);
    W.dense0 = take(2L * m * m); // [A | I] ping-pong of a coarsest level above 32 rows
    W.dense1 = take(2L * m * m);
    if (S.lean && !S.resInv)
        S.resInv = W.dense1;
    if (mixed) {
        W.ph = W.s = W.sh = W.t = W.rh = nullptr;
        W.xa = W.xb = W.rr = W.amgVec = W.amgVal = nullptr;
    }
    KW<double> &K = S.K64;
    K.d = W.d;
    K.aW = W.aW;
    K.aE = W.aE;
    K.aS = W.aS;
    K.aN = W.aN;
    K.rd = W.rd;
    K.r = W.r;
    K.rh = W.rh;
    K.pv = W.pv;
    K.v = W.v;
    K.s = W.s;
    K.t = W.t;
    K.ph = W.ph;
    K.sh = W.sh;
    K.z = W.z;
    K.xa = W.xa;
    K.xb = W.xb;
    K.rr = W.rr;
    K.x = nullptr;
    K.amgVal = W.amgVal;
    K.amgVec = W.amgVec;
}

// Locals shared by the phase functions (read from the CTA's shared state).
#define RQ_PRELUDE                                                                              \
    const DevClass &C = S.C;                                                                    \
    const Work &W = S.W;                                                                        \
    const DevSettings &st = C.st;                                                               \
    const int n = C.n, nx = C.nx, ny = C.ny, nfy = C.nfy;                                       \
    const double nu = C.nu;                                                                     \
    const double sk1 = S.coeff[0], sw1 = S.coeff[1], b1 = S.coeff[2], al1 = S.coeff[3];         \
    const double sk2 = S.coeff[4], sw2 = S.coeff[5], b2 = S.coeff[6], al2 = S.coeff[7];         \
    const double bs = S.coeff[8], a1 = S.coeff[9];                                              \
    auto blend = [](double p1, double p2, double F1) { return F1 * p1 + (1.0 - F1) * p2; };    \
    (void)st; (void)n; (void)nx; (void)ny; (void)nfy; (void)nu; (void)sk1; (void)sw1;          \
    (void)b1; (void)al1; (void)sk2; (void)sw2; (void)b2; (void)al2; (void)bs; (void)a1;         \
    (void)blend;

// ---------------------------------------------------------------- phases
// Each phase is a barrier-free sweep over cells or faces; the caller places
// the barriers and reductions. Phases are separate (non-inlined) functions so
// every sweep gets its own register allocation.
__device__ __noinline__ void phInitCells(Shared &S) {
    RQ_PRELUDE
    const double U0 = C.init[0], U1 = C.init[1], P0 = C.init[3], K0 = C.init[4], W0 = C.init[5];
    FOR_CELLS(c) {
        W.Ux[c] = U0;
        W.Uy[c] = U1;
        W.p[c] = P0;
        W.k[c] = K0;
        const double y = dmax(C.wd[c], 1e-20);
        const double om = dmax((C.balance ? 6.0 : 60.0) * C.nu / (b1 * y * y), W0);
        W.w[c] = om;
        W.F1[c] = 1.0;
        W.F2[c] = 1.0;
        W.Pk[c] = 0.0;
        W.CD[c] = 0.0;
        W.nuT[c] = a1 * K0 / dmax(a1 * om, 1e-20);
        W.S[c] = 0.0;
    }
}

// A cached converged state (fields layout, 11 x n) in place of the uniform one; the
// strain starts from zero as in solve() (SIMPLESolver.cpp:1205).
__device__ __noinline__ void phInitWarm(Shared &S, const double *wf) {
    RQ_PRELUDE
    FOR_CELLS(c) {
        W.Ux[c] = wf[c];
        W.Uy[c] = wf[n + c];
        W.p[c] = wf[3 * n + c];
        W.k[c] = wf[4 * n + c];
        W.w[c] = wf[5 * n + c];
        W.nuT[c] = wf[6 * n + c];
        W.F1[c] = wf[7 * n + c];
        W.F2[c] = wf[8 * n + c];
        W.Pk[c] = wf[9 * n + c];
        W.CD[c] = wf[10 * n + c];
        W.S[c] = 0.0;
    }
}

// interpolated flux of the velocity (ux, uy given at owner o and neighbour q) through face f
__device__ __forceinline__ double faceFlux(const DevClass &C, int f, int o, int q, const double *ux,
                                           const double *uy) {
    const double w = __ldg(C.fw + f);
    const double x = ux[o] * w + ux[q] * (1.0 - w), y = uy[o] * w + uy[q] * (1.0 - w);
    return x * __ldg(C.fsx + f) + y * __ldg(C.fsy + f);
}

__device__ __noinline__ void phInitFlux(Shared &S) {
    RQ_PRELUDE
    FOR_OWN(f, n + nfy) {
        int o, q;
        W.phi[f] = faceCells(C, f, o, q) ? faceFlux(C, f, o, q, W.Ux, W.Uy) : 0.0;
    }
}

// Iteration start: the velocity to compare against, and the gradients of U, p and (on a
// turbulence update) k and omega from one load of the cell's geometry. One CTA of a 384-cell
// class spends its time here on issuing instructions, not on data: with the geometry formed
// per field and two divisions per gradient this phase took 10 800 cycles.
__device__ __noinline__ void phStart(Shared &S, bool turbUpdate) {
    RQ_PRELUDE
    const double iBeta = 1.0 / S.wallBeta;
    FOR_CELLS(c) {
        const Cell q = cellOf(C, c);
        const GradGeo G(C, q);
        double gx, gy;
        W.Uxp[c] = W.Ux[c];
        W.Uyp[c] = W.Uy[c];
        G.of(q, nx, W.Ux, 0.0, 0.0, gx, gy);
        W.gUxx[c] = gx;
        W.gUxy[c] = gy;
        G.of(q, nx, W.Uy, 0.0, 0.0, gx, gy);
        W.gUyx[c] = gx;
        W.gUyy[c] = gy;
        const double pc = W.p[c]; // pressure wall faces carry the owner value (Neumann)
        G.of(q, nx, W.p, pc, pc, gx, gy);
        W.gPx[c] = gx;
        W.gPy[c] = gy;
        if (turbUpdate) {
            G.of(q, nx, W.k, 0.0, 0.0, gx, gy);
            W.gKx[c] = gx;
            W.gKy[c] = gy;
            G.of(q, nx, W.w, q.south ? 0.0 : __ldg(C.wallFw + q.i) * iBeta,
                 q.north ? 0.0 : __ldg(C.wallFw + nx + q.i) * iBeta, gx, gy);
            W.gWx[c] = gx;
            W.gWy[c] = gy;
        }
    }
}

__device__ __noinline__ void phClosure(Shared &S, double floorV) {
    RQ_PRELUDE
            FOR_CELLS(c) {
                const double s11 = W.gUxx[c], s22 = W.gUyy[c];
                const double s12 = 0.5 * (W.gUxy[c] + W.gUyx[c]);
                const double Sc = sqrt(2.0 * (s11 * s11 + s22 * s22 + 0.0 + 2.0 * (s12 * s12 + 0.0 + 0.0)));
                W.S[c] = Sc;
                const double kc = dmax(W.k[c], 0.0), wc = dmax(W.w[c], 1e-20);
                const double y = dmax(C.wd[c], 1e-20);
                const double cd = 2.0 * sw2 / wc * (W.gKx[c] * W.gWx[c] + W.gKy[c] * W.gWy[c]);
                W.CD[c] = cd;
                const double sqk = sqrt(dmax(kc, 0.0)), ws = dmax(wc, 1e-20);
                const double ys = dmax(y, 1e-20), y2 = ys * ys;
                const double t1 = sqk / (bs * ws * ys);
                const double t2 = 500.0 * nu / (y2 * ws);
                const double t3 = 4.0 * sw2 * kc / (dmax(cd, 1e-10) * y2);
                const double arg1 = dmin(dmax(t1, t2), t3);
                const double F1 = tanh(arg1 * arg1 * arg1 * arg1);
                W.F1[c] = F1;
                const double u1 = 2.0 * t1;
                const double arg2 = dmax(u1, t2);
                const double F2 = tanh(arg2 * arg2);
                W.F2[c] = F2;
                double den = dmax(a1 * wc, Sc * F2);
                den = dmax(den, 1e-20);
                const double nut = a1 * kc / den;
                const double raw = nut * Sc * Sc;
                const double lim = 10.0 * bs * dmax(kc, 0.0) * dmax(wc, 1e-20);
                W.Pk[c] = dmin(raw, lim);
                W.nuT[c] = dmax(nut, floorV);
            }
}

// gradient of the solved Ux for the y assembly (Uy, and so its gradient from
// phStart, is unchanged until the y solve)
__device__ __noinline__ void phGradU(Shared &S) {
    RQ_PRELUDE
    FOR_CELLS(c) {
        const Cell q = cellOf(C, c);
        const GradGeo G(C, q);
        double gx, gy;
        G.of(q, nx, W.Ux, 0.0, 0.0, gx, gy);
        W.gUxx[c] = gx;
        W.gUxy[c] = gy;
    }
}

// The internal faces of the momentum assembly, each once (assembleMomentum
// :303-482): the diffusion coefficient D = nu_f A / delta (both components: stored
// by the x pass in pCoeff, free until the p' assembly), the transpose-stress flux of
// this component (phiPred, free likewise) and its limitedLinearUpwind deferred
// correction (fScr, :495-532). Wall faces belong to one cell and are formed by the cell
// sweep.
__device__ __noinline__ void phMomentumFaces(Shared &S, int comp) {
    RQ_PRELUDE
    const double *U = comp == 0 ? W.Ux : W.Uy;
    const double *gUx = comp == 0 ? W.gUxx : W.gUyx; // grad of this component
    const double *gUy = comp == 0 ? W.gUxy : W.gUyy;
    const double *colX = comp == 0 ? W.gUxx : W.gUxy; // dUx/dx_comp
    const double *colY = comp == 0 ? W.gUyx : W.gUyy; // dUy/dx_comp
    const double *nuT = W.nuT, *phi = W.phi;
    double *D = W.pCoeff, *ts = W.phiPred, *cc = W.fScr;
    FOR_OWN(f, n + nfy) {
        int o, q;
        if (!faceCells(C, f, o, q))
            continue;
        const double w = __ldg(C.fw + f), v = 1.0 - w, F = phi[f];
        const double cf = w * nuT[o] + v * nuT[q];
        const double gxf = colX[o] * w + colX[q] * v, gyf = colY[o] * w + colY[q] * v;
        const int up = F > 0.0 ? o : q;
        const double corr = limitedCorr(F, U[q] - U[o], gUx[up], gUy[up], __ldg(C.fdx + f),
                                        __ldg(C.fdy + f));
        if (comp == 0)
            D[f] = (nu + cf) * __ldg(C.fad + f);
        ts[f] = cf * (gxf * __ldg(C.fsx + f) + gyf * __ldg(C.fsy + f));
        cc[f] = corr;
    }
}

// The momentum rows of one component from the face values of phMomentumFaces (a resolved
// wall: molecular viscosity, U_b = 0, no flux), summed in the reference's order (x faces, y
// faces, walls); the row's residual. The x pass leaves V / a_P in aP for the p' equation.
__device__ __noinline__ void phMomentum(Shared &S, int comp, int rp) {
    RQ_PRELUDE
    const double *U = comp == 0 ? W.Ux : W.Uy, *gP = comp == 0 ? W.gPx : W.gPy;
    const double *phi = W.phi, *D = W.pCoeff, *tsf = W.phiPred, *ccf = W.fScr;
    const double fb = comp == 0 ? st.fx : st.fy;
    double acc[3];
    parkOver(acc, S, rp, n, [&](int c) {
        const Cell q = cellOf(C, c);
        const int fW = q.W, fE = c, fS = n + c, fN = n + c + nx;
        const double FW = phi[fW], FE = phi[fE], DW = D[fW], DE = D[fE];
        double aS = 0.0, aN = 0.0, dS, dN, ts = tsf[fE] - tsf[fW], cc = ccf[fW] - ccf[fE];
        if (q.south) {
            const double F = phi[fS], d = D[fS];
            dS = d + dmax(-F, 0.0);
            aS = -(d + dmax(F, 0.0));
            ts -= tsf[fS];
            cc += ccf[fS];
        } else {
            dS = nu * __ldg(C.fad + fS);
        }
        if (q.north) {
            const double F = phi[fN], d = D[fN];
            dN = d + dmax(F, 0.0);
            aN = -(d + dmax(-F, 0.0));
            ts += tsf[fN];
            cc -= ccf[fN];
        } else {
            dN = nu * __ldg(C.fad + fN);
        }
        const double aW = -(DW + dmax(FW, 0.0)), aE = -(DE + dmax(-FE, 0.0));
        double dsum = (DW + dmax(-FW, 0.0)) + (DE + dmax(FE, 0.0));
        dsum = q.south ? (dsum + dS) + dN : (dsum + dN) + dS; // the wall comes last
        const double V = __ldg(C.vol + c), Uc = U[c];
        double bsum = -(gP[c] * V);
        if (fb != 0.0)
            bsum += fb * V;
        bsum += ts;
        bsum += cc;
        bsum += C.relax[0] * dsum * Uc; // (1 - alpha) / alpha
        const double dd = dsum * C.relax[1];
        if (comp == 0) {
            W.aP[c] = fabs(dd) > 1e-30 ? V / dd : 0.0;
            const double uy = W.Uy[c];
            acc[2] += dsum * sqrt(Uc * Uc + uy * uy);
        }
        W.d[c] = dd;
        W.aW[c] = aW;
        W.aE[c] = aE;
        W.aS[c] = aS;
        W.aN[c] = aN;
        W.b[c] = bsum;
        // residual b - A U of this row (relaxation cancels at U)
        const double tS = q.south ? aS * U[c - nx] : 0.0, tN = q.north ? aN * U[c + nx] : 0.0;
        const double rc = bsum - accum4(q, dd * Uc, aW * U[q.W], aE * U[q.E], tS, tN);
        W.r[c] = rc;
        acc[0] += fabs(rc);
        acc[1] += rc * rc;
    });
}

// Predicted face flux (stored Rhie-Chow, :1401-1419) and the coefficient of p'. The flux of
// the velocity at the iteration start is interpolated here, beside the new one, from the
// same geometry (a sweep of its own in phStart cost a store and ten loads per face).
__device__ __noinline__ void phPressureFaces(Shared &S, int rp) {
    RQ_PRELUDE
    const double relaxCorr = 1.0 - st.aU;
    const double *Ux = W.Ux, *Uy = W.Uy, *Uxp = W.Uxp, *Uyp = W.Uyp, *dP = W.aP, *p = W.p;
    const double *gPx = W.gPx, *gPy = W.gPy, *phi = W.phi;
    double *pred = W.phiPred, *coeff = W.pCoeff;
    double fs[1];
    parkOver(fs, S, rp, n + nfy, [&](int f) {
        int o, q;
        double ph = 0.0, pc = 0.0;
        if (faceCells(C, f, o, q)) {
            const double w = __ldg(C.fw + f), v = 1.0 - w, sx = __ldg(C.fsx + f),
                         sy = __ldg(C.fsy + f), ad = __ldg(C.fad + f);
            const double x = Ux[o] * w + Ux[q] * v, y = Uy[o] * w + Uy[q] * v;
            const double x0 = Uxp[o] * w + Uxp[q] * v, y0 = Uyp[o] * w + Uyp[q] * v;
            const double dF = w * dP[o] + v * dP[q];
            const double gbx = gPx[o] * w + gPx[q] * v, gby = gPy[o] * w + gPy[q] * v;
            ph = x * sx + y * sy;
            ph -= dF * ((p[q] - p[o]) * ad - (gbx * __ldg(C.fex + f) + gby * __ldg(C.fey + f)));
            ph += relaxCorr * (phi[f] - (x0 * sx + y0 * sy));
            pc = dF * ad;
        }
        pred[f] = ph;
        coeff[f] = pc;
        fs[0] += fabs(ph);
    });
}

__device__ __noinline__ void phPressureCells(Shared &S, int rp) {
    RQ_PRELUDE
        double pacc[2];
        parkOver(pacc, S, rp, n, [&](int c) {
            const Cell q = cellOf(C, c);
            const int fE = c, fW = q.W, fN = n + c + nx, fS = n + c;
            // diagonal: coefficients of internal faces in order
            const double cW = W.pCoeff[fW], cE = W.pCoeff[fE];
            const double cS = q.south ? W.pCoeff[fS] : 0.0, cN = q.north ? W.pCoeff[fN] : 0.0;
            double dsum = 0.0;
            {
                const double x1 = q.xEfirst ? cE : cW, x2 = q.xEfirst ? cW : cE;
                dsum = dsum + x1;
                dsum = dsum + x2;
                if (q.yNfirst) {
                    if (q.north)
                        dsum = dsum + cN;
                } else {
                    if (q.south)
                        dsum = dsum + cS;
                    if (q.north)
                        dsum = dsum + cN;
                }
            }
            // source: -(owner fluxes) + (neighbour fluxes), walls last
            const double tW = W.phiPred[fW], tE = -W.phiPred[fE];
            double bsum = 0.0;
            {
                const double x1 = q.xEfirst ? tE : tW, x2 = q.xEfirst ? tW : tE;
                bsum += x1;
                bsum += x2;
                if (q.yNfirst) {
                    bsum += -W.phiPred[fN];
                    bsum += -W.phiPred[fS]; // bottom wall
                } else {
                    bsum += q.south ? W.phiPred[fS] : -W.phiPred[fS];
                    bsum += -W.phiPred[fN];
                }
            }
            if (c == 0)
                dsum += fabs(dsum) > 1e-30 ? dsum : 1.0; // pin of the outlet-free system
            W.d[c] = dsum;
            W.aW[c] = -cW;
            W.aE[c] = -cE;
            W.aS[c] = -cS;
            W.aN[c] = -cN;
            W.b[c] = bsum;
            W.r[c] = bsum;
            W.pp[c] = 0.0;
            pacc[0] += fabs(bsum);
            pacc[1] += bsum * bsum;
        });
}

// Pressure-velocity corrections (:916-940, :1443-1467): U -= grad p' V / aP with
// owner-valued wall faces for grad p', p += alpha_p p', the face fluxes from p'; on a
// turbulence update also the k and omega values the change norms compare against.
// The k and omega gradients of the transport equations are the ones phStart formed:
// k and omega do not change between the start of the iteration and their solves.
__device__ __noinline__ void phCorrect(Shared &S, bool turbUpdate) {
    RQ_PRELUDE
    const double *pp = W.pp;
    FOR_CELLS(c) {
        const Cell q = cellOf(C, c);
        const GradGeo G(C, q);
        double gx, gy;
        const double pc = pp[c], dP = W.aP[c]; // V / a_P
        G.of(q, nx, pp, pc, pc, gx, gy);
        W.Ux[c] -= dP * gx;
        W.Uy[c] -= dP * gy;
        W.p[c] += st.aP * pc;
        if (turbUpdate) {
            W.kOld[c] = W.k[c];
            W.wOld[c] = W.w[c];
        }
    }
    const double *pred = W.phiPred, *coeff = W.pCoeff;
    double *phi = W.phi;
    FOR_OWN(f, n + nfy) {
        int o, q;
        phi[f] = faceCells(C, f, o, q) ? pred[f] - coeff[f] * (pp[q] - pp[o]) : 0.0;
    }
}

// bounds of the solved k and omega (:1489, :1505-1513); a wall cell of omega takes its wall
// value
__device__ __forceinline__ void clampK(const Shared &S, int c) {
    const DevSettings &st = S.C.st;
    S.W.k[c] = dmax(st.kMin, dmin(st.kMax, S.W.k[c]));
}
__device__ __forceinline__ double clampW(const Shared &S, int c, double iB1) {
    const DevClass &C = S.C;
    const Cell q = cellOf(C, c);
    double v = dmax(C.st.wMin, dmin(1e15, S.W.w[c]));
    if (!q.south || !q.north)
        v = __ldg(C.wallW + wallSlot(C, q)) * iB1;
    S.W.w[c] = v;
    return v;
}

// The internal faces of the k or omega assembly, each once (assembleKEquation
// :947-1028, assembleOmegaEquation :1030-1171): the diffusion coefficient
// (nu + sigma(F1_f) nuT)_f A / delta (pCoeff), the deferred correction of the
// limitedLinearUpwind face value (fScr, addConvectionCorrection :495-552) and, for
// omega with the near-wall balance, its face term (phiPred, :1073-1087). Wall faces
// are formed by the cell sweep.
__device__ __noinline__ void phTurbFaces(Shared &S, int eq) {
    RQ_PRELUDE
    const double *X = eq == 0 ? W.k : W.w;
    const double *gX = eq == 0 ? W.gKx : W.gWx, *gY = eq == 0 ? W.gKy : W.gWy;
    const double s1 = eq == 0 ? sk1 : sw1, s2 = eq == 0 ? sk2 : sw2;
    const bool balance = eq == 1 && C.balance;
    const double amp = balance ? 6 * nu / b1 : 0.0;
    const double *nuT = W.nuT, *F1 = W.F1, *phi = W.phi;
    double *D = W.pCoeff, *bal = W.phiPred, *cc = W.fScr;
    FOR_OWN(f, n + nfy) {
        int o, q;
        if (!faceCells(C, f, o, q))
            continue;
        const double w = __ldg(C.fw + f), v = 1.0 - w, F = phi[f];
        const double sg = blend(s1, s2, w * F1[o] + v * F1[q]);
        const double et = sg * (w * nuT[o] + v * nuT[q]); // the turbulent part
        const int up = F > 0.0 ? o : q;
        const double corr =
            limitedCorr(F, X[q] - X[o], gX[up], gY[up], __ldg(C.fdx + f), __ldg(C.fdy + f));
        D[f] = (nu + et) * __ldg(C.fad + f);
        if (balance) // singular near-wall balance (:1073-1087)
            bal[f] = amp * (et * __ldg(C.fb1 + f) - (nu + et) * __ldg(C.fb2 + f));
        cc[f] = corr;
    }
}

// The k or omega rows from the face values of phTurbFaces (the wall faces here),
// sources, relaxation and the omega wall constraint (constrainOmega :687-704), summed in
// face order, and the residual of the constrained initial guess: a wall cell of omega holds
// its wall value, its row is decoupled and its neighbours take the value to their right-hand
// side, so no row reads a wall cell's unknown and it is set here. (The residual as a sweep
// of its own re-read the five coefficients: 3300 cycles at 384 cells, 8700 at 1536.)
__device__ __noinline__ void phTurbAssemble(Shared &S, int eq, int rp) {
    RQ_PRELUDE
    double *X = eq == 0 ? W.k : W.w;
    const double *phi = W.phi, *D = W.pCoeff, *bal = W.phiPred, *ccf = W.fScr;
    const double s1 = eq == 0 ? sk1 : sw1, s2 = eq == 0 ? sk2 : sw2;
    const bool balance = eq == 1 && C.balance;
    const double iB1 = 1.0 / b1, iBeta = 1.0 / S.wallBeta;
    double acc[1];
    parkOver(acc, S, rp, n, [&](int c) {
        if (eq == 1) // the bounds of the k just solved (read below at this cell only)
            clampK(S, c);
        const Cell q = cellOf(C, c);
        const int fW = q.W, fE = c, fS = n + c, fN = n + c + nx;
        const double F1 = W.F1[c], nuT = W.nuT[c];
        const double FW = phi[fW], FE = phi[fE], DW = D[fW], DE = D[fE];
        const double wall = nu + blend(s1, s2, F1) * nuT; // viscosity at a wall face
        double aW = -(DW + dmax(FW, 0.0)), aE = -(DE + dmax(-FE, 0.0)), aS = 0.0, aN = 0.0;
        double dS, dN, bsum = 0.0, bl = 0.0, cc = ccf[fW] - ccf[fE];
        if (balance)
            bl = bal[fE] - bal[fW];
        if (q.south) {
            const double F = phi[fS], d = D[fS];
            dS = d + dmax(-F, 0.0);
            aS = -(d + dmax(F, 0.0));
            cc += ccf[fS];
            if (balance)
                bl -= bal[fS];
        } else {
            dS = wall * __ldg(C.fad + fS);
            if (eq == 1)
                bsum += dS * (__ldg(C.wallFw + q.i) * iBeta);
        }
        if (q.north) {
            const double F = phi[fN], d = D[fN];
            dN = d + dmax(F, 0.0);
            aN = -(d + dmax(-F, 0.0));
            cc -= ccf[fN];
            if (balance)
                bl += bal[fN];
        } else {
            dN = wall * __ldg(C.fad + fN);
            if (eq == 1)
                bsum += dN * (__ldg(C.wallFw + nx + q.i) * iBeta);
        }
        double dsum = (DW + dmax(-FW, 0.0)) + (DE + dmax(FE, 0.0));
        dsum = q.south ? (dsum + dS) + dN : (dsum + dN) + dS; // the wall comes last
        const double V = __ldg(C.vol + c), wc = dmax(W.w[c], 1e-20);
        if (eq == 0) {
            bsum += W.Pk[c] * V;
            dsum += bs * wc * V;
        } else {
            const double Sv = W.S[c];
            const double lim = 10.0 * bs * dmax(W.k[c], 0.0) * wc / dmax(nuT, 1e-30);
            bsum += blend(al1, al2, F1) * dmin(Sv * Sv, lim) * V;
            dsum += blend(b1, b2, F1) * wc * V;
            bsum += (1.0 - F1) * W.CD[c] * V;
            if (balance) {
                const double corr = bl + nu * (6 * nu * iB1) * __ldg(C.slap + c) * V;
                if (corr < 0)
                    dsum -= corr / wc;
                else
                    bsum += corr;
            }
        }
        bsum += cc;
        const double xo = X[c];
        bsum += C.relax[2 + 2 * eq] * dsum * xo; // (1 - alpha) / alpha
        dsum *= C.relax[3 + 2 * eq];
        double rc;
        if (eq == 1 && (!q.south || !q.north)) {
            const double val = __ldg(C.wallW + wallSlot(C, q)) * iB1;
            aW = aE = aS = aN = 0.0;
            bsum = dsum * val;
            X[c] = val;
            rc = 0.0;
        } else {
            if (eq == 1 && q.j == 1) {
                bsum -= aS * (__ldg(C.wallW + q.i) * iB1);
                aS = 0.0;
            }
            if (eq == 1 && q.j == ny - 2) {
                bsum -= aN * (__ldg(C.wallW + nx + q.i) * iB1);
                aN = 0.0;
            }
            const double tS = q.south && !(eq == 1 && q.j == 1) ? aS * X[c - nx] : 0.0;
            const double tN = q.north && !(eq == 1 && q.j == ny - 2) ? aN * X[c + nx] : 0.0;
            rc = bsum - accum4(q, dsum * xo, aW * X[q.W], aE * X[q.E], tS, tN);
        }
        W.d[c] = dsum;
        W.aW[c] = aW;
        W.aE[c] = aE;
        W.aS[c] = aS;
        W.aN[c] = aN;
        W.b[c] = bsum;
        W.r[c] = rc;
        acc[0] += rc * rc;
    });
}

// Change norms; mx[4], mx[5]: squares of the largest |U| and |dU|.
__device__ __noinline__ void phNorms(Shared &S, bool turbUpdate, double (&mx)[6]) {
    RQ_PRELUDE
    if (turbUpdate && threadIdx.x == 0)
        S.wallBeta = b1;
    const double iB1 = 1.0 / b1;
    FOR_CELLS(c) {
        if (turbUpdate) {
            const double w = clampW(S, c, iB1), k = W.k[c];
            mx[0] = dmax(mx[0], fabs(k));
            mx[1] = dmax(mx[1], fabs(w));
            mx[2] = dmax(mx[2], fabs(k - W.kOld[c]));
            mx[3] = dmax(mx[3], fabs(w - W.wOld[c]));
        }
        const double x = W.Ux[c], y = W.Uy[c], ax = x - W.Uxp[c], ay = y - W.Uyp[c];
        mx[4] = dmax(mx[4], x * x + y * y);
        mx[5] = dmax(mx[5], ax * ax + ay * ay);
    }
}

__device__ __noinline__ void phProbes(Shared &S) {
    RQ_PRELUDE
            if (threadIdx.x < C.nobs) { // PreparedObservation::evaluate (:678-772)
                const int t = threadIdx.x;
                const int cell = C.pcell[t];
                const double *X = C.obsComp == 0 ? W.Ux : W.Uy;
                const double center = X[cell];
                double bx = 0, by = 0;
                for (int k = 0; k < C.pnnb[t]; ++k) {
                    const int nb = C.pnb[4 * t + k];
                    const double diff = (nb < 0 ? 0.0 : X[nb]) - center;
                    bx += C.pwt[4 * t + k] * C.pdx[4 * t + k] * diff;
                    by += C.pwt[4 * t + k] * C.pdy[4 * t + k] * diff;
                }
                double gx = 0.0, gy = 0.0;
                if (fabs(C.pdet[t]) > 1e-14 * (C.paxx[t] * C.payy[t] + 1e-300)) {
                    gx = (C.payy[t] * bx - C.paxy[t] * by) / C.pdet[t];
                    gy = (C.paxx[t] * by - C.paxy[t] * bx) / C.pdet[t];
                }
                S.q[t] = center + gx * C.pox[t] + gy * C.poy[t];
            }
}

__device__ void runSolve(Shared &S, const DevJob &job) {
    const DevClass &C = S.C;
    const Work &W = S.W;
    const DevSettings &st = C.st;
    const int n = C.n, nx = C.nx, ny = C.ny, nfy = C.nfy;
    const double nu = C.nu;
    int rp = 0;
    // coefficients (InferenceParameterSet order) and their blends (SSTModel.hpp:12-61)
    const double sk1 = S.coeff[0], sw1 = S.coeff[1], b1 = S.coeff[2], al1 = S.coeff[3];
    const double sk2 = S.coeff[4], sw2 = S.coeff[5], b2 = S.coeff[6], al2 = S.coeff[7];
    const double bs = S.coeff[8], a1 = S.coeff[9];
    auto blend = [](double p1, double p2, double F1) { return F1 * p1 + (1.0 - F1) * p2; };
    const double inf = __longlong_as_double(0x7ff0000000000000LL);

    // ---- initUniform (SIMPLESolver.cpp:267-298) and applyAllBCs, or the cached state of
    // a warm start (ForwardModel.cpp:79-82), whose turbulence is established
    if (job.warm)
        phInitWarm(S, job.warm);
    else
        phInitCells(S);
    if (threadIdx.x < 4)
        S.cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0)
        S.wallBeta = job.warm ? job.warmBeta : C.beta1Init;
    if (threadIdx.x == 0) {
        S.haveQPrev = 0;
        S.innerKrylov = 0;
        S.innerPressure = 0;
        for (int t = 0; t < 8; ++t)
            S.stage[t] = 0;
        S.tmark = clock64();
    }
    SYNC();
    // phi = interpolated fluxes of the initial state (wall faces carry U_b = 0)
    phInitFlux(S);
    SYNC();

    // the loop state lives in shared memory (LoopState); every thread writes the same
    // values, and reads after its own writes
    LoopState &Ls = S.L;
    bool &established = Ls.established, &converged = Ls.converged, &diverged = Ls.diverged;
    int &amgNeed = Ls.amgNeed, &amgAfter = Ls.amgAfter; // AMG coarse-value refresh state
    double &lastK = Ls.lastK, &lastW = Ls.lastW;
    double &worst = Ls.worst, &fluxRef = Ls.fluxRef, &n0x = Ls.n0x, &n0y = Ls.n0y, &n0p = Ls.n0p;
    int &status = Ls.status, &finalIter = Ls.finalIter;
    double &rateU = Ls.rateU;
    established = job.warm != nullptr;
    amgNeed = 1;
    amgAfter = -1;
    lastK = 1.0;
    lastW = 1.0;
    worst = inf;
    fluxRef = 0.0;
    n0x = n0y = n0p = 1.0;
    status = 1;
    finalIter = st.maxIter;
    converged = diverged = false;
    rateU = __longlong_as_double(0x7ff8000000000000LL);


    for (int iter = 0; iter < st.maxIter; ++iter) {
        const bool turbActive = iter >= st.turbStart;
        const bool turbUpdate = turbActive && ((iter - st.turbStart) % st.turbInterval == 0);
        // ---- phase: save U, interpolated old flux, gradients of U and p
        phStart(S, turbUpdate);
        SYNC();

        mark(S, 7);
        // ---- SST closure (SSTModel.cpp:157-241) and the startup nuT floor (:1322-1337)
        if (turbUpdate) {
            if (!established && iter >= st.turbStart + st.floorIters)
                established = true;
            const double floorV = established ? 0.0 : 0.1 * nu;
            phClosure(S, floorV);
            SYNC();
        }

        mark(S, 1);
        // ---- momentum x then y (assembleMomentum :303-482)
        LinRes *resU = Ls.resU;
        double &momRes = Ls.momRes, &momScale = Ls.momScale;
        for (int comp = 0; comp < 2; ++comp) {
            if (comp == 1) { // gradients of the updated Ux for the y assembly
                phGradU(S);
                SYNC();
            }
            double *U = comp == 0 ? W.Ux : W.Uy;
            double acc[3];
            phMomentumFaces(S, comp);
            SYNC();
            phMomentum(S, comp, rp);
            totalSums(acc, S, rp);
            momRes = comp == 0 ? acc[0] : dmax(momRes, acc[0]);
            if (comp == 0)
                momScale = acc[2];
            solveBicg(S, rp, U, sqrt(acc[1]), st.innerIter, st.innerTol, &resU[comp]);
            if (threadIdx.x == 0)
                S.innerKrylov += resU[comp].iterations;
            SYNC();
        }

        mark(S, 2);
        // ---- predicted flux (stored Rhie-Chow, :1401-1419) and p' assembly (:717-830)
        double fs[1], pacc[2];
        phPressureFaces(S, rp);
        totalSums(fs, S, rp);
        phPressureCells(S, rp);
        totalSums(pacc, S, rp);
        Ls.contScaled = pacc[0] / dmax(fs[0], 1e-300);
        Ls.fluxScale = fs[0];
        mark(S, 3);
        LinRes &resP = Ls.resP;
        resP = solvePressure(S, rp, W.pp, sqrt(pacc[1]), st.innerIter, st.innerTol, st.pSolver,
                             amgNeed, amgAfter);
        if (threadIdx.x == 0)
            S.innerPressure += resP.iterations;
        SYNC();

        mark(S, 4);
        // ---- corrections (:916-940, :1443-1467)
        phCorrect(S, turbUpdate);
        SYNC();

        // ---- turbulence (:1476-1538)
        LinRes &resK = Ls.resK, &resW = Ls.resW;
        resK = LinRes{0, 0, 0, true};
        resW = LinRes{0, 0, 0, true};
        if (turbUpdate) {
            // the clamp of k runs inside the omega assembly and the clamp of omega
            // inside the change norms (each reads only its own cell's value)
            for (int eq = 0; eq < 2; ++eq) { // 0: k, 1: omega
                double *X = eq == 0 ? W.k : W.w;
                double acc[1];
                phTurbFaces(S, eq);
                SYNC();
                phTurbAssemble(S, eq, rp);
                totalSums(acc, S, rp);
                LinRes &rr = eq == 0 ? resK : resW;
                solveBicg(S, rp, X, sqrt(acc[0]), st.innerIter, st.innerTol, &rr);
                if (threadIdx.x == 0)
                    S.innerKrylov += rr.iterations;
                SYNC();
            }
        }

        mark(S, 6);
        // ---- change norms and bookkeeping (:1520-1715)
        double mx[6] = {1e-30, 1e-30, 0.0, 0.0, 0.0, 0.0};
        phNorms(S, turbUpdate, mx);
        blockMax<6>(mx, S, rp);
        if (turbUpdate) {
            lastK = mx[2] / mx[0];
            lastW = mx[3] / mx[1];
        }
        Ls.uChange = sqrt(mx[5]) / dmax(sqrt(mx[4]), 1e-300);
        // one barrier pair for every sample of this iteration (U, k, omega, monitor)
        SYNC();
        if (threadIdx.x == 0) {
            S.ring[0][S.cnt[0] % kWindowCap] = Ls.uChange;
            S.cnt[0] += 1;
            if (turbUpdate) {
                S.ring[1][S.cnt[1] % kWindowCap] = lastK;
                S.cnt[1] += 1;
                S.ring[2][S.cnt[2] % kWindowCap] = lastW;
                S.cnt[2] += 1;
            }
        }
        SYNC();
        const bool haveMonitor = C.nobs > 0;
        if (haveMonitor && iter % (st.monitorInterval > 1 ? st.monitorInterval : 1) == 0) {
            phProbes(S);
            SYNC();
            bool finite = true;
            for (int t = 0; t < C.nobs; ++t)
                finite = finite && isfinite(S.q[t]);
            if (!finite) { // the reference throws here: the row becomes Unknown
                status = 4;
                finalIter = iter;
                break;
            }
            if (S.haveQPrev) {
                double qMax = 0.0, dq = 0.0;
                for (int t = 0; t < C.nobs; ++t)
                    qMax = dmax(qMax, fabs(S.q[t]));
                for (int t = 0; t < C.nobs; ++t) {
                    const double fl = C.obsFloor[t];
                    dq = dmax(dq, fabs(S.q[t] - S.qPrev[t]) / dmax(dmax(fabs(S.q[t]), fl), 1e-300));
                }
                pushSample(S, 3, dq);
            }
            SYNC();
            if (threadIdx.x < C.nobs)
                S.qPrev[threadIdx.x] = S.q[threadIdx.x];
            if (threadIdx.x == 0)
                S.haveQPrev = 1;
            SYNC();
        }
        // the history entry of this iteration (ResidualEntry order); no phase call follows
        const double tol = st.tol, negligible = 0.01 * tol;
        double e[11];
        e[0] = iter;
        e[1] = resU[0].initialRes;
        e[2] = resU[1].initialRes;
        e[3] = 0.0;
        e[4] = resP.initialRes;
        e[5] = turbActive ? lastK : 0.0;
        e[6] = turbActive ? lastW : 0.0;
        e[7] = momRes / dmax(momScale, 1e-300);
        e[8] = Ls.contScaled;
        e[9] = Ls.uChange;
        e[10] = inf;
        if (iter == 0) {
            n0x = dmax(e[1], 1e-30);
            n0y = dmax(e[2], 1e-30);
            n0p = dmax(e[4], 1e-30);
            fluxRef = Ls.fluxScale;
        } else if (iter < 50) {
            n0p = dmax(n0p, e[4]);
            fluxRef = dmax(fluxRef, Ls.fluxScale);
        }
        auto safe = [](double v, double ref) { return ref < 1e-20 ? 0.0 : v / ref; };
        const double nm = dmax(n0x, n0y);
        const double nUx = safe(e[1], nm), nUy = safe(e[2], nm);
        const double nP = safe(e[4], dmax(n0p, fluxRef));
        double maxRes = dmax(dmax(nUx, nUy), nP);
        if (turbActive)
            maxRes = dmax(dmax(maxRes, lastK), lastW);
        bool bad = !isfinite(lastK) || !isfinite(lastW);
        for (int t = 1; t <= 9; ++t)
            bad = bad || !isfinite(e[t]);
        if (bad)
            maxRes = inf;
        // The contraction estimates only change the verdict when every directly
        // measured quantity already passes, so they are evaluated then, on the
        // last iteration, on a divergence exit and for recorded history.
        const double qLast = (haveMonitor && S.cnt[3] > 0) ? S.ring[3][(S.cnt[3] - 1) % kWindowCap] : inf;
        double cheap = dmax(dmax(e[7], e[8]), e[9]);
        if (turbActive)
            cheap = dmax(dmax(cheap, lastK), lastW);
        if (haveMonitor)
            cheap = dmax(cheap, qLast);
        const bool divergingNow = isnan(maxRes) || isinf(maxRes) || maxRes > st.divLimit;
        const bool needEst = cheap < tol || iter == st.maxIter - 1 || divergingNow ||
                             (job.hist && iter < job.histCap);
        double w;
        if (needEst) {
            const Est eU = estimate(S, 0, st.window, negligible);
            e[10] = eU.remaining;
            rateU = eU.rate;
            double wv = e[7];
            wv = dmax(wv, e[8]);
            wv = dmax(wv, e[9]);
            wv = dmax(wv, e[10]);
            if (turbActive) {
                const Est eK = estimate(S, 1, st.window, negligible);
                const Est eW = estimate(S, 2, st.window, negligible);
                wv = dmax(wv, lastK);
                wv = dmax(wv, eK.remaining);
                wv = dmax(wv, lastW);
                wv = dmax(wv, eW.remaining);
            }
            if (haveMonitor) {
                const Est eQ = estimate(S, 3, st.window, negligible);
                wv = dmax(wv, qLast);
                wv = dmax(wv, eQ.remaining);
            }
            w = isfinite(wv) ? wv : inf;
        } else {
            w = cheap; // >= tol: not a verdict iteration
        }
        if (job.hist && iter < job.histCap && threadIdx.x == 0)
            for (int t = 0; t < 11; ++t)
                job.hist[11L * iter + t] = e[t];
        if (bad)
            w = inf;
        worst = w;
        const bool turbScheduled = st.turbStart < st.maxIter;
        if (w < tol && iter > 0 && (!turbScheduled || (turbActive && established))) {
            converged = true;
            finalIter = iter;
            status = 0;
            break;
        }
        if (isnan(maxRes) || isinf(maxRes) || maxRes > st.divLimit) {
            diverged = true;
            finalIter = iter;
            status = 2;
            break;
        }
    }
    SYNC();
    const bool stalled = !converged && !diverged && status == 1 && isfinite(rateU) && rateU >= 1.0;

    // ---- outputs: verdict, probe predictions, log-likelihood (ObservationOperator.hpp:592-609)
    if (status == 0 || status == 1) {
        phProbes(S);
        SYNC();
    }
    if (threadIdx.x == 0) {
        RowOut o;
        o.iterations = finalIter;
        o.stalled = stalled;
        o.converged = converged;
        o.finalWorst = worst;
        o.contractionRate = rateU;
        o.status = status;
        o.loglik = status == 2 ? -1e6 : (status == 4 ? -1e6 : 0.0);
        if (status == 0 || status == 1) {
            double ll = 0.0;
            bool ok = true;
            for (int t = 0; t < C.nobs; ++t) {
                const double v = S.q[t];
                job.pred[t] = v;
                ok = ok && isfinite(v);
                const double diff = v - C.obsVal[t];
                ll += -0.5 * diff * diff / C.obsVar[t];
            }
            if (!ok || !isfinite(ll)) {
                o.status = 4;
                o.loglik = -1e6;
            } else {
                o.loglik = ll;
            }
        }
        if (o.status != 0 && o.status != 1)
            for (int t = 0; t < C.nobs; ++t)
                job.pred[t] = __longlong_as_double(0x7ff8000000000000LL);
        *job.row = o;
    }
    if (job.fields && status != 2) {
        const double *src[11] = {W.Ux, W.Uy, nullptr, W.p, W.k, W.w, W.nuT, W.F1, W.F2, W.Pk, W.CD};
        for (int b = 0; b < 11; ++b)
            FOR_CELLS(c) job.fields[(long)b * n + c] = src[b] ? src[b][c] : 0.0;
    } else if (job.fields) { // a diverged solve leaves no valid state (ForwardModel.cpp:88-96)
        for (long e = gTid(); e < 11L * n; e += gThreads())
            job.fields[e] = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (job.snap && status != 2) {
        FOR_OWN(f, n + nfy)
            job.snap[f] = W.phi[f];
        if (threadIdx.x == 0) {
            job.snap[n + nfy] = S.wallBeta;
            job.snap[n + nfy + 1] = established ? 1.0 : 0.0;
        }
    }
    SYNC();
}

} // namespace

// One job on this CTA: class descriptor into shared memory, admission and unpack
// of theta (InferenceParameterSet::inBounds / unpack), the solve or the
// InvalidParameters row, then the per-row timing record.
__device__ void runJob(Shared &S, const DevJob &job, double *ws, double *arena, int arenaDoubles) {
    long long t0 = 0;
    if (threadIdx.x == 0)
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    {
        const int words = sizeof(DevClass) / 4;
        const int *src = reinterpret_cast<const int *>(job.cls);
        int *dst = reinterpret_cast<int *>(&S.C);
        for (int t = threadIdx.x; t < words; t += blockDim.x)
            dst[t] = src[t];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        bool ok = true;
        for (int i = 0; i < 11; ++i)
            S.coeff[i] = S.C.base[i];
        for (int a = 0; a < S.C.nActive; ++a) {
            const int idx = S.C.active[a];
            const double v = job.theta[a];
            if (v < S.C.lo[idx] || v > S.C.hi[idx] || isnan(v) || isinf(v))
                ok = false;
            S.coeff[idx] = v;
        }
        S.admitted = ok;
        S.slices = kCluster ? solveSlices(S.C.n) : 1;
        S.ownSlices = S.slices / ctaCount();
        if (ok)
            carve(S, ws, arena, arenaDoubles);
    }
    __syncthreads();
    if (S.admitted && S.lean)
        resTables(S);
    if (S.admitted) {
        runSolve(S, job);
    } else {
        if (threadIdx.x == 0) {
            const double nan = __longlong_as_double(0x7ff8000000000000LL);
            RowOut o{3, 0, 0, 0, -1e30, nan, nan};
            *job.row = o;
        }
        for (int t = threadIdx.x; t < S.C.nobs; t += blockDim.x)
            job.pred[t] = __longlong_as_double(0x7ff8000000000000LL);
        if (job.fields)
            for (long e = gTid(); e < 11L * S.C.n; e += gThreads())
                job.fields[e] = __longlong_as_double(0x7ff8000000000000LL);
    }
    __syncthreads();
    if (gTid() == 0 && job.clock) {
        long long t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        job.clock[0] = t0;
        job.clock[1] = t1;
        job.clock[2] = S.admitted ? S.innerKrylov : 0;
        job.clock[3] = S.admitted ? S.innerPressure : 0;
        for (int t = 0; t < 8; ++t)
            job.clock[4 + t] = S.admitted ? S.stage[t] : 0;
    }
}

__device__ __forceinline__ long long globalNs() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Resident CTAs that the register budget of a CTA size is set for (128 registers at 512
// threads and 256, 168 below, 80 at 768, 64 at 1024). Said explicitly because ptxas may
// otherwise halve the budget of the 512-thread kernels to fit two on an SM, which costs a
// 384-cell solve 45 % (spills in every phase).
constexpr int ctasPerSM(int nt) { return nt >= 512 ? 1 : nt == 256 ? 2 : nt == 128 ? 3 : 6; }

// One kernel body, instantiated per CTA size so each gets its full register budget.
template <int NT, bool Cluster>
__global__ void __launch_bounds__(NT, ctasPerSM(NT)) solveKernel(const DevJob *jobs, int njobs, int *nextJob,
                                                  double *wsBase, long wsStride, int arenaDoubles) {
    extern __shared__ __align__(16) unsigned char smemRaw[];
    Shared &S = *reinterpret_cast<Shared *>(smemRaw);
    double *arena = reinterpret_cast<double *>(smemRaw + kSharedBytes);
    double *ws = wsBase + wsStride * (blockIdx.x / ctaCount());
    if constexpr (kCluster)
        SYNC(); // every CTA of the cluster has started: its shared memory can be written
    for (;;) {
        if constexpr (kCluster) {
            if (gTid() == 0) {
                const int j = atomicAdd(nextJob, 1);
                for (int r = 0; r < ctaCount(); ++r)
                    putRemote(&S.job, j, r);
            }
        } else if (threadIdx.x == 0) {
            S.job = atomicAdd(nextJob, 1);
        }
        SYNC();
        const int j = S.job;
        if (j >= njobs)
            break;
        runJob(S, jobs[j], ws, arena, arenaDoubles);
        // an inadmissible draw passes no cluster barrier in runJob: without this one rank 0
        // could store the next job into a CTA whose warps have not read the last one
        if constexpr (kCluster)
            SYNC();
    }
}

// The serving loop: persistent CTAs claim requests as the host publishes them.
// Requests live in host-mapped memory (ServeQueue); a CTA claims request h only
// once h < published, by a compare-and-swap on the device-side head, so no
// ticket is ever held for an unpublished request. A CTA leaves when the host
// closes the queue and nothing is left, or after idleNs without work (the host
// launches more CTAs when requests wait and fewer than the slots run); closed = 2
// cancels the requests not yet claimed (solves in flight still finish). A request
// solves in its own pool region when it carries one (DevJob::ws), else in the CTA's
// slot workspace. Results go straight to host-mapped rows; the request's done flag
// is raised after a system-scope fence; every CTA counts its exit.
template <int NT, bool Cluster>
__global__ void __launch_bounds__(NT, ctasPerSM(NT)) serveKernel(ServeQueue q, double *wsBase, long wsStride,
                                                  int arenaDoubles) {
    extern __shared__ __align__(16) unsigned char smemRaw[];
    Shared &S = *reinterpret_cast<Shared *>(smemRaw);
    double *arena = reinterpret_cast<double *>(smemRaw + kSharedBytes);
    double *ws = wsBase + wsStride * blockIdx.x;
    for (;;) {
        if (threadIdx.x == 0) {
            int got = -1;
            const long long idleFrom = globalNs();
            for (;;) {
                int closed, pub;
                asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(closed) : "l"(q.closed) : "memory");
                if (closed >= 2) // cancelled: leave unclaimed requests alone
                    break;
                asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(pub) : "l"(q.published) : "memory");
                pub = min(pub, q.capacity);
                const int h = atomicAdd(q.head, 0);
                if (h < pub) {
                    if (atomicCAS(q.head, h, h + 1) == h) {
                        got = h;
                        break;
                    }
                    continue;
                }
                if (closed) // closed and drained
                    break;
                if (globalNs() - idleFrom > q.idleNs) // idle: leave (the host tops up)
                    break;
                __nanosleep(4000);
            }
            S.job = got;
            if (got >= 0)
                S.jd = q.jobs[got];
        }
        __syncthreads();
        const int j = S.job;
        if (j < 0)
            break;
        runJob(S, S.jd, S.jd.ws ? S.jd.ws : ws, arena, arenaDoubles);
        __threadfence_system();
        __syncthreads();
        if (threadIdx.x == 0)
            asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(q.done + j), "r"(1) : "memory");
        __syncthreads();
    }
    if (threadIdx.x == 0) // counted so the host can tell how many CTAs still run
        atomicAdd(q.exits, 1);
}

// ---------------------------------------------------------------- allocation-free single solve
// One job passed by value (no job array, no queue counter), solved by one CTA or cluster in
// the scratch array.
template <int NT, bool Cluster>
__global__ void __launch_bounds__(NT, ctasPerSM(NT)) solveOneKernel(DevJob job, double *ws, int arenaDoubles) {
    extern __shared__ __align__(16) unsigned char smemRaw[];
    Shared &S = *reinterpret_cast<Shared *>(smemRaw);
    double *arena = reinterpret_cast<double *>(smemRaw + kSharedBytes);
    if (threadIdx.x == 0)
        S.jd = job;
    __syncthreads();
    runJob(S, S.jd, ws, arena, arenaDoubles);
}

// The kernels of one CTA size. This file is compiled once per CTA size with RQ_CTA set
// (the phases are separate functions that ptxas allocates for each kernel's register
// budget, so one object for all sizes would compile serially), and once without for the
// host entry points.
enum SolveEntry { kEntrySolve = 0, kEntryServe = 1, kEntryOne = 2, kEntryBytes = 3 };
constexpr int kClusterThreads = 768; // CTA size of the cluster kernels
template <int NT, bool Cluster> void *solveEntry(int kind);

#ifdef RQ_CTA
template <> void *solveEntry<RQ_CTA, kCluster>(int kind) {
    switch (kind) {
    case kEntrySolve: return reinterpret_cast<void *>(&solveKernel<RQ_CTA, kCluster>);
#if RQ_CTA >= 256 && !defined(RQ_CLUSTER)
    case kEntryServe: return reinterpret_cast<void *>(&serveKernel<RQ_CTA, kCluster>);
#endif
    case kEntryOne: return reinterpret_cast<void *>(&solveOneKernel<RQ_CTA, kCluster>);
    case kEntryBytes: return reinterpret_cast<void *>(kSharedBytes);
    default: return nullptr;
    }
}
#else
template <> void *solveEntry<64, false>(int);
template <> void *solveEntry<128, false>(int);
template <> void *solveEntry<256, false>(int);
template <> void *solveEntry<512, false>(int);
template <> void *solveEntry<768, false>(int);
template <> void *solveEntry<1024, false>(int);
template <> void *solveEntry<kClusterThreads, true>(int);

// Workspace of rq_evaluate_noalloc: one solve's scratch in a fixed device array
// that the module owns, so that the call itself needs no device allocation. It
// lives on every GPU that loads this library until the process exits.
constexpr long kNoAllocScratchDoubles = 1L << 20; // 8 MiB
static __device__ __align__(256) double g_noallocScratch[kNoAllocScratchDoubles];

size_t solveSharedBytes() { return kSharedBytes; }
size_t clusterSharedBytes() {
    return reinterpret_cast<size_t>(solveEntry<kClusterThreads, true>(kEntryBytes));
}
long residentDoubles(const DevClass &C, int block) {
    if (C.st.precision != kFP64 || block > kResMaxThreads || C.n > kResCells * block)
        return 0;
    return resExchange(C.n) + (C.resAmg ? (C.amgVecs + 31) / 32 * 32 : 0);
}

namespace {
void *entryOf(int kind, int block) {
    switch (block) {
    case 64: return solveEntry<64, false>(kind);
    case 128: return solveEntry<128, false>(kind);
    case 256: return solveEntry<256, false>(kind);
    case 512: return solveEntry<512, false>(kind);
    case 768: return solveEntry<768, false>(kind);
    case 1024: return solveEntry<1024, false>(kind);
    default: return nullptr;
    }
}
void *pick(int block) { return entryOf(kEntrySolve, block); }
void *pickServe(int block) { return entryOf(kEntryServe, block); }
// the function of a launch shape, and its dynamic shared memory
void *shapeEntry(int kind, const LaunchShape &sh) {
    if (sh.cluster > 0)
        return sh.block == kClusterThreads ? solveEntry<kClusterThreads, true>(kind) : nullptr;
    return entryOf(kind, sh.block);
}
size_t shapeBytes(const LaunchShape &sh) {
    return (sh.cluster > 0 ? clusterSharedBytes() : solveSharedBytes()) +
           sizeof(double) * static_cast<size_t>(sh.arenaDoubles);
}
// The limits are set to the device's own, not to the launch's: they belong to the function, and
// another thread may be launching it with another arena.
cudaError_t setAttributes(void *fn) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    return e;
}
cudaLaunchConfig_t configOf(const LaunchShape &sh, int solves, cudaStream_t stream,
                            cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(solves * (sh.cluster > 1 ? sh.cluster : 1));
    cfg.blockDim = dim3(sh.block);
    cfg.dynamicSmemBytes = shapeBytes(sh);
    cfg.stream = stream;
    if (sh.cluster > 1) {
        attr->id = cudaLaunchAttributeClusterDimension;
        attr->val.clusterDim.x = sh.cluster;
        attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cfg;
}
} // namespace

bool launchVariantExists(int block) { return pick(block) != nullptr; }

int normalizeBlock(int block) {
    return block <= 64 ? 64 : block <= 128 ? 128 : block <= 256 ? 256 : block <= 512 ? 512
         : block <= 768 ? 768 : 1024;
}

cudaError_t launchSolve(const DevJob *jobs, int njobs, int *nextJob, double *ws, long wsStride,
                        int solves, const LaunchShape &sh, cudaStream_t stream) {
    void *fn = shapeEntry(kEntrySolve, sh);
    if (!fn)
        return cudaErrorInvalidConfiguration;
    cudaError_t e = setAttributes(fn);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = configOf(sh, solves, stream, &attr);
    int arenaDoubles = sh.arenaDoubles;
    void *args[] = {&jobs, &njobs, &nextJob, &ws, &wsStride, &arenaDoubles};
    e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess)
        return e;
    return cudaGetLastError();
}

int concurrentSolves(const LaunchShape &sh, int sms) {
    void *fn = shapeEntry(kEntrySolve, sh);
    if (!fn || setAttributes(fn) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int count = 0;
    if (sh.cluster > 1) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = configOf(sh, sms, nullptr, &attr);
        if (cudaOccupancyMaxActiveClusters(&count, fn, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return count;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&count, fn, sh.block, shapeBytes(sh)) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return count * sms;
}

cudaError_t launchServe(const ServeQueue &q, double *ws, long wsStride, int grid, int block,
                        int arenaDoubles, cudaStream_t stream) {
    const size_t smem = solveSharedBytes() + sizeof(double) * static_cast<size_t>(arenaDoubles);
    void *fn = pickServe(block);
    if (!fn)
        return cudaErrorInvalidConfiguration;
    cudaError_t e = setAttributes(fn);
    if (e != cudaSuccess)
        return e;
    ServeQueue qq = q;
    void *args[] = {&qq, &ws, &wsStride, &arenaDoubles};
    e = cudaLaunchKernel(fn, dim3(grid), dim3(block), args, smem, stream);
    if (e != cudaSuccess)
        return e;
    return cudaGetLastError();
}

int serveBlocksPerSM(int block, int arenaDoubles) {
    const size_t smem = solveSharedBytes() + sizeof(double) * static_cast<size_t>(arenaDoubles);
    void *fn = pickServe(block);
    if (!fn || setAttributes(fn) != cudaSuccess)
        return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, block, smem) != cudaSuccess)
        return 0;
    return blocks;
}

long noAllocScratchDoubles() { return kNoAllocScratchDoubles; }

// The device address of the scratch array on the current device. The host-side name
// of a __device__ array is only a stand-in, not an address a kernel may use, so it is
// looked up with cudaGetSymbolAddress (no allocation; the first lookup on a device
// loads the module there). Callers resolve it once per handle, when the handle is
// created, so that nothing stale survives a device reset.
cudaError_t noAllocScratch(double **out) {
    double *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_noallocScratch);
    if (e != cudaSuccess)
        return e;
    *out = p;
    return cudaSuccess;
}

cudaError_t launchSolveNoAlloc(const DevJob &job, double *scratch, const LaunchShape &sh,
                               cudaStream_t stream) {
    if (!scratch)
        return cudaErrorInvalidDevicePointer;
    double *ws = scratch;
    void *fn = shapeEntry(kEntryOne, sh);
    if (!fn)
        return cudaErrorInvalidConfiguration;
    cudaError_t e = setAttributes(fn);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = configOf(sh, 1, stream, &attr);
    DevJob j = job;
    int arenaDoubles = sh.arenaDoubles;
    void *args[] = {&j, &ws, &arenaDoubles};
    e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess)
        return e;
    return cudaGetLastError();
}

#endif // RQ_CTA

} // namespace rq
