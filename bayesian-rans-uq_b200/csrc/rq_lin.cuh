// Device-side layout of the standalone batched linear solves (rq_linsolve.cu):
// one DevLinSys per LDU system, its matrices and hierarchy in HBM, its vectors
// in the workspace slot of the CTA that solves it.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace rq {

constexpr int kLinMaxLevels = 16;
constexpr int kLinThreads = 1024;
constexpr int kLinSmallThreads = 512; // of the systems of one slice
constexpr int kLinMaxSlices = 16;   // slices of a system's sums: the CTAs of its largest cluster
constexpr int kLinMaxLocalBytes = 208 * 1024; // shared memory of the local levels' vectors
constexpr int kLinLocalRows = 2048; // rows of a level that every CTA of a cluster runs whole
enum LinKind : int32_t { kLinAmg = 0, kLinPcg = 1, kLinBicgstab = 2 };

// SolverResult (core/include/LinearSolver.hpp:137-143); the layout of rq_solver_result
struct LinOut {
    int32_t iterations, converged;
    double finalRes, initialRes;
};

struct DevLinLevel {
    int32_t n, nc;                   // rows; rows of the next level (0 on the coarsest)
    int64_t vecOff;                  // b, x, r of this level in the level-vector area (levels
                                     // 1 .. loc - 1) or in a CTA's shared memory (loc and above)
    // Rows (level 0: diagonal, then faces in face order; above: column order) in slices of
    // 1 << sh rows, 32 of them (a warp's loads of entry k are consecutive) or, where equal
    // widths would more than double the entries, one (plain CSR): entry k of row i is at
    // ptr[i >> sh] + (k << sh) + (i & ((1 << sh) - 1)); padding has column -1.
    int32_t sh, pad;
    const int32_t *ptr, *col;
    const double *val, *rdg;         // values, 1/diag
    const float *val32, *rdg32;      // FP32 copies (mixed form)
    const int32_t *agg;              // row -> next-level row
    const int32_t *childPtr, *childIdx; // next-level row -> rows, ascending
};

struct DevLinSys {
    int32_t n, nlev, kind, precision, maxIter, m; // m: rows of the coarsest level
    int32_t loc;      // first level (>= 1) of at most kLinLocalRows rows
    int32_t slices;   // slices of its sums: a multiple of the CTAs that solve it
    double tol;
    int64_t lvOff;    // doubles: FP64 level vectors (after 8n FP64 Krylov vectors)
    int64_t f32Off;   // doubles: start of the FP32 area (mixed form)
    int64_t lvOff32;  // floats from f32Off: FP32 level vectors (after 6n FP32 vectors)
    const double *b;
    double *x;        // initial guess in, solution out
    const double *inv;
    const float *inv32;
    LinOut *out;
    DevLinLevel lev[kLinMaxLevels];
};

// Threads of a CTA (kLinThreads or kLinSmallThreads), CTAs per system, and shared memory of the
// local levels' vectors.
struct LinShape {
    int threads = kLinThreads, cluster = 1;
    size_t localBytes = 0;
};
// Persistent clusters, one system at a time each; *next zeroed by the caller; ws: `slots`
// workspaces of wsStride doubles, one per cluster.
cudaError_t launchLinear(const DevLinSys *systems, int nsys, int *next, double *ws, long wsStride,
                         int slots, const LinShape &shape, cudaStream_t stream);
// Clusters that run at once (0: the shape does not fit).
int linConcurrent(const LinShape &shape);

} // namespace rq
