// Launch entry points of the device code (rq_solver.cu), used by rq_capi.cu.
#pragma once
#include <cuda_runtime.h>

#include "rq_device.cuh"

namespace rq {

size_t solveSharedBytes();   // fixed shared memory of a CTA
size_t clusterSharedBytes(); // the same of the cluster kernels
// Doubles at the start of the arena that the resident inner solvers of a class need in CTAs
// of `block` threads (0: they do not apply, rq_resident.cuh).
long residentDoubles(const DevClass &C, int block);
// Launch shape of a solve: CTA size (64, 128, 256, 512, 768 or 1024), shared-memory arena
// per CTA in doubles for the hot arrays (0 = all global), and the CTAs per solve of the cluster
// kernels (768 threads; the arena holds the small AMG levels), 0: the kernels of one CTA.
struct LaunchShape {
    int block, arenaDoubles, cluster;
};
// Slices of the sums of a class that the cluster kernels solve: the CTAs of its largest
// cluster, whatever the number it runs on.
constexpr int kMaxSlices = 8;
#ifdef __CUDACC__
__host__ __device__
#endif
inline int solveSlices(int n) { return n < 32768 ? 4 : kMaxSlices; }
// Persistent solves: each pulls job indices from *nextJob (zeroed by the caller)
// until njobs are taken; ws is solves x wsStride doubles of per-solve workspace.
cudaError_t launchSolve(const DevJob *jobs, int njobs, int *nextJob, double *ws, long wsStride,
                        int solves, const LaunchShape &sh, cudaStream_t stream);
// Solves of the shape that run at once on a GPU of `sms` SMs (0: does not fit).
int concurrentSolves(const LaunchShape &sh, int sms);
bool launchVariantExists(int block);
// The serving loop (serveKernel): grid persistent CTAs of `block` threads (256, 512
// or 1024) serving q until it is closed and drained, or until q.idleNs passes
// without a request.
cudaError_t launchServe(const ServeQueue &q, double *ws, long wsStride, int grid, int block,
                        int arenaDoubles, cudaStream_t stream);
int serveBlocksPerSM(int block, int arenaDoubles);
int normalizeBlock(int block);
// One solve of one job in the module's fixed scratch array (no device allocation):
// capacity in doubles, the array's device address on the current device (looked up
// by cudaGetSymbolAddress at every call of noAllocScratch, which allocates nothing),
// and the launch (one solve of the given shape) on that address.
long noAllocScratchDoubles();
cudaError_t noAllocScratch(double **out);
cudaError_t launchSolveNoAlloc(const DevJob &job, double *scratch, const LaunchShape &sh,
                               cudaStream_t stream);
// Posterior weights (rq_stats.cu): one CTA; out = {max, sum of exp, non-finite count}.
cudaError_t launchWeights(const double *ll, const double *lq, int64_t n, double *w, double *out,
                          cudaStream_t stream);
// Statistics of an ensemble (rq_stats.cu), each with numpy's rounding: multinomial
// indices for given uniforms (cdf: n doubles of scratch), column mean / variance,
// the k-th smallest nonnegative value, |a - b|, and test -/+ radius.
cudaError_t launchResample(const double *w, int64_t n, const double *u, int64_t m, int64_t *idx,
                           double *cdf, cudaStream_t stream);
cudaError_t launchMoments(const double *x, int64_t n, int d, double *mean, double *var,
                          cudaStream_t stream);
cudaError_t launchSelect(const double *v, int64_t n, int64_t k, double *out, cudaStream_t stream);
cudaError_t launchAbsDiff(const double *a, const double *b, int64_t n, double *out,
                          cudaStream_t stream);
cudaError_t launchInterval(const double *test, int64_t m, const double *radius, double *lo,
                           double *hi, cudaStream_t stream);

} // namespace rq
