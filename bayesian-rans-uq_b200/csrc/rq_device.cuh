// Device-side data layout of the B200 forward model. One mesh class (mesh,
// boundary conditions, viscosity, settings, probes, AMG pattern) lives in HBM
// once; every coefficient draw is a job that one CTA (or one thread-block cluster) runs from cold start to
// its verdict without leaving the GPU (see rq_solver.cu).
#pragma once
#include <cstddef>
#include <cstdint>

namespace rq {

constexpr int kMaxLevels = 12;    // AMG levels (the reference allows 20; meshes here need <= 8)
constexpr int kLocalRows = 1536;  // rows of an AMG level that every CTA of a cluster runs whole
constexpr int kMaxCoarse = 128;   // rows of the dense coarsest AMG level
constexpr int kMaxProbes = 64;    // observations per problem
constexpr int kWindowCap = 64;    // 2 * convergenceWindow samples kept per estimator

enum Precision : int32_t { kFP64 = 0, kMixed = 1 };
enum PSolver : int32_t { kPAmg = 0, kPPcg = 1, kPBicgstab = 2 };

// SolverSettings subset of the hot path (rans-uq FlowFields.hpp:70-241).
struct DevSettings {
    int32_t maxIter, innerIter, window, monitorInterval;
    int32_t turbStart, turbInterval, floorIters, pSolver;
    int32_t precision, pad;
    double tol, innerTol, divLimit;
    double aU, aP, aK, aW;
    double fx, fy;
    double kMin, kMax, wMin;
};

// Levels >= 1 are stored in ELL form in slices of 32 rows: entry k of row i, in column
// order, is at slot ellRow(i, width) + 32 k (a warp reading entry k of 32 consecutive rows
// touches consecutive addresses, and the entries of a row lie at constant distances, which
// the load instructions hold as immediates); shorter rows and the rows that fill the last
// slice are padded with column -1. The transfer operators between level l and level l+1
// (nc rows) are ELL too: the prolongation P (entry k of fine row i: its k-th coarse row and
// the weight) and the restriction P^T (entry k of coarse row I: its k-th fine row and the
// weight), padded with -1.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int ellRow(int i, int width) {
    return (i >> 5) * (width << 5) + (i & 31);
}
struct DevAmgLevel {
    int32_t n, nnz;             // rows; value slots (levels >= 1)
    int32_t valOff, vecOff;     // per-solve value / vector offsets (levels >= 1)
    int32_t width, pad;         // ELL width (levels >= 1)
    int32_t pw, rw;             // prolongation / restriction ELL widths (all but the last level)
    const int32_t *ecol, *diagPos;       // ELL columns (-1: padding); slot of the diagonal
    const int32_t *pcol, *rcol;          // prolongation / restriction ELL columns
    const double *pval, *rval;           // and weights
    const uint16_t *ecol16, *pcol16, *rcol16; // the same columns in 16 bits, padding as column
                                              // 0 (its values are 0); classes with resAmg
    const int32_t *gPtr, *gSrc;          // next-level value slot -> entries of this level
    const double *gW;                    // each entry's weight P_iI P_jJ in the Galerkin sum
};

struct DevClass {
    int32_t nx, ny, n, nfy;
    int32_t balance, nobs, nlev, obsComp;
    double nu, beta1Init;      // beta1 of the initial wall-omega face value (applyAllBCs default)
    double init[6];            // U xyz, p, k, omega
    DevSettings st;
    // cells
    const double *vol, *ivol, *wd; // volume, 1 / volume (1 where it is below 1e-30), wall distance
    // faces (x faces 0 .. n-1, then y faces): owner weight, area vector, A / delta, A times
    // the unit vector along d, d = owner-to-neighbour vector
    const double *fw, *fsx, *fsy, *fad, *fex, *fey, *fdx, *fdy;
    // wall columns (bottom, then top): 60 nu / y^2 of the omega wall face value and
    // (6 or 60) nu / y^2 of the wall cell value (resolvedWallOmega), both to be divided by beta1
    const double *wallFw, *wallW;
    // planar singular omega balance: A times the singular gradient and A times the
    // difference quotient per face, the singular Laplacian per cell
    const double *fb1, *fb2, *slap;
    // (1 - alpha) / alpha and 1 / alpha of U, k and omega
    double relax[6];
    // probes: 4 neighbour slots each
    const int32_t *pcell, *pnnb, *pnb;
    const double *pox, *poy, *paxx, *paxy, *payy, *pdet, *pdx, *pdy, *pwt;
    const double *obsVal, *obsVar, *obsFloor;
    DevAmgLevel lev[kMaxLevels];
    double amgW, amgAlpha;     // V-cycle smoother weight, coarse-correction scale
    int32_t amgVals, amgVecs;  // per-solve doubles for coarse values / vectors
    int32_t resAmg;            // the 16-bit columns are set: coarseRes runs the FP64 V-cycle
    int32_t locLevel, locDoubles; // first level of at most kLocalRows rows (cluster solves run
                                  // it and the coarser ones per CTA), and their vectors
    int32_t amgSweeps;   // damped-Jacobi sweeps before and after each coarse correction
    int64_t wsDoubles;         // per-solve workspace
    // InferenceParameterSet: active indices, the coefficients filling the rest,
    // and the admission bounds (core/include/InferenceParameters.hpp:67-77, 127-165)
    int32_t nActive, pad2;
    int32_t active[11], pad3;
    double base[11], lo[11], hi[11];
};

// Outcome of one draw; the status values and order follow EvaluationStatus
// (core/include/EvaluationTypes.hpp:6).
struct RowOut {
    int32_t status, iterations, stalled, converged;
    double loglik, finalWorst, contractionRate;
};

struct DevJob {
    const DevClass *cls;
    const double *theta; // nActive values of this draw (device)
    RowOut *row;
    double *pred;      // nobs
    double *fields;    // optional 11 x n
    double *hist;      // optional hist_cap x 11
    long long *clock;  // optional, 12 per row: global-timer ns at start and end, inner
                       // Krylov iterations, inner pressure iterations, 8 stage cycle counts
    int32_t histCap;
    int32_t pad;
    // Warm start (optional): a converged state in the fields layout (11 x n: Ux Uy Uz p k
    // omega nuT F1 F2 Pk CDkw) copied in place of the uniform initial state, and the beta1
    // its wall-face omega was last set with (the cached solve's own coefficient).
    const double *warm;
    double warmBeta;
    // Snapshot (optional, written with the fields): the n + nfy face fluxes in the
    // device face layout (x faces, then y faces), the beta1 of the final wall-face omega,
    // and the turbulence-established marker (0 or 1).
    double *snap;
    // Solve workspace of this job (the serving loop's pool region of the job's class),
    // or null: the CTA's own per-slot workspace.
    double *ws;
};

// Request queue of the serving loop. The host appends requests (jobs[i], with
// theta, row and prediction slots) to host-mapped memory and then raises
// *published; CTAs claim them in order through *head (device memory) and raise
// done[i] when request i's results are in place.
struct ServeQueue {
    const DevJob *jobs;      // host-mapped, capacity entries
    const int *published;    // host-mapped: requests published so far
    const int *closed;       // host-mapped: 1 = no more requests (drain), 2 = cancel the rest
    int *done;               // host-mapped: one flag per request
    int *head;               // device: next request to claim
    int *exits;              // device: CTAs that have left (idle, drained or cancelled)
    int capacity, pad;
    long long idleNs;
};

} // namespace rq
