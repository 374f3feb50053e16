// C ABI of the standalone linear solves (rq_linear_solve*, rq_linsys_*): host
// set-up of the LDU systems (rq_linsys.cpp), their packing into device buffers
// and the persistent linKernel launch (rq_linsolve.cu).
#include "rq_capi_common.h"

#include <functional>
#include <queue>

using namespace rqc;

// Standalone LDU systems resident on the device (rq_linsys_*).
struct rq_linsys {
    int nsys = 0, kind = 0, precision = 0, maxLevels = 0;
    // systems of one launch shape: a range of `sys`, the clusters launched for it with a
    // workspace each, and a stream beside the caller's (all but the first group)
    struct Group {
        int first = 0, count = 0, slots = 1;
        long wsStride = 0, wsOff = 0;
        rq::LinShape shape;
        cudaStream_t stream = nullptr;
        cudaEvent_t done = nullptr;
    };
    std::vector<Group> groups;
    cudaEvent_t fork = nullptr;
    ~rq_linsys() {
        for (Group &g : groups) {
            if (g.done)
                cudaEventDestroy(g.done);
            if (g.stream)
                cudaStreamDestroy(g.stream);
        }
        if (fork)
            cudaEventDestroy(fork);
    }
    int64_t totalRows = 0, totalNnz = 0;
    std::vector<int> rows;
    std::vector<int64_t> xOff;
    std::vector<rq::DevLinSys> sys; // queue order (groups, each largest first), device pointers
    DevBuf dI, dD, dF, dB, dX, dSys, dOut, dWs, dNext;
    std::mutex mu;
};

namespace {

void checkSolveArgs(int maxIter, double tol) {
    if (maxIter < 0 || !std::isfinite(tol) || tol <= 0.)
        throw std::invalid_argument("linear solve requires matching x, nonnegative iteration "
                                    "cap and positive finite tolerance");
}

// Slices of a system's sums, and so the CTAs of its largest cluster: the smallest power of two
// that leaves a thread fewer than two rows, at most 16.
int linSlices(int rows) {
    int c = 1;
    while (c < rq::kLinMaxSlices && 2L * c * rq::kLinThreads <= rows)
        c *= 2;
    return c;
}

// Threads per CTA, by the rows alone: 512 with 128 registers for the systems of one slice, else
// 1024 with 64. Measured on a B200, ms of FP64 AMG solves, 1 / 592 systems of n x n, 512 against
// 1024 threads: n = 16 0.24 / 1.00 against 0.30 / 1.31, n = 24 0.32 / 1.33 against 0.37 / 1.64,
// n = 32 0.44 / 2.02 against 0.57 / 2.56, n = 45 1.00 / 4.34 against 1.01 / 4.49.
int linThreads(int rows) { return linSlices(rows) == 1 ? rq::kLinSmallThreads : rq::kLinThreads; }

// How often the clusters of a batch are halved from their largest size (no bit of a result
// depends on it): the number for which a list of the systems, largest first, ends first on a
// GPU of which a cluster of c CTAs takes one part in clustersAtOnce(c). A solve takes about
// 3860 (rows / 4096)^0.3 + rows / c units of time (0.35 us), up to 2.4 times that as the rows
// in flight outgrow L2. Measured on a B200, ms of FP64 AMG solves to 1e-10, by halvings 0 / 1 /
// 2 / 3 / 4 (systems of n x n):
//     1 of 64    1.48 / 1.67 /  1.87            148 of  64    7.21 /  3.51 /  2.95
//     1 of 128   2.13 / 2.33 /  3.0 / 4.4 / 6.5  32 of 128   10.7 /  6.9 /  4.2 /  5.9 /  8.9
//                                               148 of 128   46.3 / 23.9 / 18.9 / 15.2 / 15.6
//     1 of 256   4.1 /  5.5 /  8.2 / 14 / 24     16 of 256   13.1 / 14.0 / 14.2 / 24.5 / 43.6
//     1 of 512  11.4 / 18.4 / 32.5 / 61 / 113    32 of 512   97 / 98 / 77 / 138 / 255
// (One 512-thread CTA per system, the former kernel: 148 of 64 about 7, 148 of 128 28.8, one of
// 512 about 260.)
template <typename AtOnce>
int linHalvings(const std::vector<int> &rowsLargestFirst, AtOnce clustersAtOnce) {
    const int most = rq::kLinMaxSlices;
    std::vector<double> share(most + 1, -1.0); // by CTAs; 0: one of kLinSmallThreads
    auto shareOf = [&](int threads, int c) {
        double &part = share[threads == rq::kLinThreads ? c : 0];
        if (part < 0.0) {
            const int k = clustersAtOnce(threads, c);
            part = k > 0 ? 1.0 / k : 2.0; // 2: does not fit
        }
        return part;
    };
    struct Run {
        double end, share, rows;
        bool operator>(const Run &o) const { return end > o.end; }
    };
    int best = -1;
    double least = 0.0;
    for (int h = 0; most >> h; ++h) {
        std::priority_queue<Run, std::vector<Run>, std::greater<Run>> running;
        double now = 0.0, free = 1.0, rows = 0.0, last = 0.0;
        bool fits = true, waits = false;
        for (int n : rowsLargestFirst) {
            const int c = std::max(1, linSlices(n) >> h);
            const double part = shareOf(linThreads(n), c);
            if (part > 1.0) {
                fits = false;
                break;
            }
            while (free < part - 1e-9) {
                now = running.top().end;
                free += running.top().share;
                rows -= running.top().rows;
                running.pop();
                waits = true;
            }
            free -= part;
            rows += n;
            const double t = 3860 * std::pow(n / 4096.0, 0.3) + static_cast<double>(n) / c;
            const double end = now + t * std::min(2.4, 1 + 0.7e-6 * rows);
            running.push({end, part, static_cast<double>(n)});
            last = std::max(last, end);
        }
        if (fits && (best < 0 || last < least)) {
            best = h;
            least = last;
        }
        if (fits && !waits) // smaller clusters only take longer
            break;
    }
    if (best < 0)
        throw RqError(RQ_E_CUDA, "linear solve kernel does not fit on an SM");
    return best;
}

void buildLinsys(rq_linsys &L, const rq_ldu *systems, int n, int kind, int precision) {
    L.nsys = n;
    L.kind = kind;
    L.precision = precision;
    for (int s = 0; s < n; ++s) {
        const rq_ldu &A = systems[s];
        rq::validateLdu(A.n_cells, A.n_faces, A.diag, A.upper, A.lower, A.source, A.owner,
                        A.neighbour);
        if (A.n_cells < 1)
            throw std::invalid_argument("linear system needs at least one cell");
    }
    // host set-up of every system, on all host threads
    std::vector<rq::LinSysHost> H(n);
    std::vector<std::string> err(n);
    std::vector<int> unsupported(n, 0);
    {
        const int nt = std::max(1, std::min<int>(n, static_cast<int>(std::thread::hardware_concurrency())));
        std::atomic<int> next{0};
        auto work = [&] {
            for (int s = next++; s < n; s = next++) {
                const rq_ldu &A = systems[s];
                try {
                    H[s] = rq::buildLinSys(A.n_cells, A.n_faces, A.diag, A.upper, A.lower, A.owner,
                                           A.neighbour, kind == rq::kLinAmg);
                } catch (const rq::LinUnsupported &e) {
                    err[s] = e.what();
                    unsupported[s] = 1;
                } catch (const std::exception &e) {
                    err[s] = e.what();
                }
            }
        };
        std::vector<std::thread> pool;
        for (int t = 1; t < nt; ++t)
            pool.emplace_back(work);
        work();
        for (auto &t : pool)
            t.join();
    }
    for (int s = 0; s < n; ++s)
        if (!err[s].empty())
            throw RqError(unsupported[s] ? RQ_E_UNSUPPORTED : RQ_E_INVALID,
                          "system " + std::to_string(s) + ": " + err[s]);
    // Layout pass: every array of every system gets an offset in one of three
    // device buffers (int32, FP64, FP32); the copies then run on all host threads.
    enum { P_PTR, P_COL, P_VAL, P_RDG, P_VAL32, P_RDG32, P_AGG, P_CPTR, P_CIDX, P_INV, P_INV32 };
    struct Piece {
        int s, l, what;
        size_t off;
        const void *src; // std::vector<int> or std::vector<double> of the host set-up
        const rq::LinLevelHost *lv; // P_COL, P_VAL, P_VAL32: the level, laid out in slices
        size_t count;
    };
    std::vector<Piece> pieces;
    size_t nI = 0, nD = 0, nF = 0;
    auto addI = [&](int s, int l, int what, const std::vector<int> &v) {
        pieces.push_back({s, l, what, nI, &v, nullptr, v.size()});
        nI += (v.size() + 7) / 8 * 8;
    };
    auto addD = [&](int s, int l, int what, const std::vector<double> &v) {
        pieces.push_back({s, l, what, nD, &v, nullptr, v.size()});
        nD += (v.size() + 3) / 4 * 4;
    };
    auto addF = [&](int s, int l, int what, const std::vector<double> &v) {
        pieces.push_back({s, l, what, nF, &v, nullptr, v.size()});
        nF += (v.size() + 7) / 8 * 8;
    };
    auto addRows = [&](int s, int l, int what, const rq::LinLevelHost &lv, size_t &total) {
        const size_t cnt = lv.slice.back();
        pieces.push_back({s, l, what, total, nullptr, &lv, cnt});
        total += (cnt + 7) / 8 * 8;
    };
    const bool mixed = precision == RQ_PREC_MIXED;
    L.rows.resize(n);
    L.xOff.resize(n);
    std::vector<rq::DevLinSys> byIndex(n);
    std::vector<long> wsOf(n);
    std::vector<size_t> localOf(n);
    for (int s = 0; s < n; ++s) {
        const rq::LinSysHost &h = H[s];
        rq::DevLinSys &d = byIndex[s];
        std::memset(&d, 0, sizeof(d));
        const int nl = static_cast<int>(h.lev.size());
        if (nl > rq::kLinMaxLevels)
            throw RqError(RQ_E_UNSUPPORTED, "AMG hierarchy deeper than 16 levels");
        d.n = h.n;
        d.nlev = nl;
        d.kind = kind;
        d.precision = mixed && kind != rq::kLinBicgstab ? 1 : 0;
        d.m = h.m;
        d.loc = nl;
        long localRows = 0; // b, x and r of the local levels fit in shared memory
        while (d.loc > 1 && h.lev[d.loc - 1].n <= rq::kLinLocalRows &&
               24 * (localRows + h.lev[d.loc - 1].n) <= rq::kLinMaxLocalBytes)
            localRows += h.lev[--d.loc].n;
        long lvecs = 0, local = 0;
        for (int l = 0; l < nl; ++l) {
            const rq::LinLevelHost &lv = h.lev[l];
            rq::DevLinLevel &dl = d.lev[l];
            dl.n = lv.n;
            dl.nc = lv.nc;
            dl.sh = lv.sh;
            long &vecs = l >= d.loc ? local : lvecs;
            dl.vecOff = l > 0 ? vecs : 0;
            if (l > 0)
                vecs += 3L * lv.n;
            addI(s, l, P_PTR, lv.slice);
            addRows(s, l, P_COL, lv, nI);
            addRows(s, l, P_VAL, lv, nD);
            addD(s, l, P_RDG, lv.rdg);
            if (d.precision) {
                addRows(s, l, P_VAL32, lv, nF);
                addF(s, l, P_RDG32, lv.rdg);
            }
            if (l + 1 < nl) {
                addI(s, l, P_AGG, lv.agg);
                addI(s, l, P_CPTR, lv.childPtr);
                addI(s, l, P_CIDX, lv.childIdx);
            }
            L.totalNnz += static_cast<int64_t>(lv.col.size());
        }
        if (kind == rq::kLinAmg) {
            addD(s, 0, P_INV, h.inv);
            if (d.precision)
                addF(s, 0, P_INV32, h.inv);
        }
        const long nn = h.n;
        d.lvOff = pad32(8 * nn);
        d.f32Off = d.lvOff + pad32(lvecs);
        d.lvOff32 = 2 * pad32((6 * nn + 1) / 2);
        const long ws = d.f32Off + (d.precision ? (d.lvOff32 / 2 + pad32((lvecs + 1) / 2)) : 0);
        wsOf[s] = ws;
        localOf[s] = static_cast<size_t>(local) * (d.precision ? sizeof(float) : sizeof(double));
        L.rows[s] = h.n;
        L.xOff[s] = L.totalRows;
        L.totalRows += h.n;
        L.maxLevels = std::max(L.maxLevels, nl);
    }
    std::unique_ptr<int32_t[]> I(new int32_t[std::max<size_t>(nI, 1)]);
    std::unique_ptr<double[]> D(new double[std::max<size_t>(nD, 1)]);
    std::unique_ptr<float[]> F(new float[std::max<size_t>(nF, 1)]);
    std::unique_ptr<double[]> hb(new double[std::max<int64_t>(L.totalRows, 1)]);
    {
        const int nt = std::max(1, std::min<int>(static_cast<int>(pieces.size()),
                                                 static_cast<int>(std::thread::hardware_concurrency())));
        std::atomic<size_t> next{0};
        std::atomic<int> nextRhs{0};
        // the entries of a level in slices: put(position, CSR entry or -1 for padding)
        auto spread = [](const rq::LinLevelHost &lv, auto put) {
            const int c = 1 << lv.sh;
            for (int i = 0; i < (lv.n + c - 1) / c * c; ++i) {
                const int at = lv.slice[i >> lv.sh], w = (lv.slice[(i >> lv.sh) + 1] - at) >> lv.sh;
                const int k0 = i < lv.n ? lv.ptr[i] : 0, len = i < lv.n ? lv.ptr[i + 1] - k0 : 0;
                for (int k = 0; k < w; ++k)
                    put(at + (k << lv.sh) + (i & (c - 1)), k < len ? k0 + k : -1);
            }
        };
        auto work = [&] {
            for (size_t k = next++; k < pieces.size(); k = next++) {
                const Piece &p = pieces[k];
                switch (p.what) {
                case P_COL:
                    spread(*p.lv, [&](int at, int e) { I[p.off + at] = e < 0 ? -1 : p.lv->col[e]; });
                    break;
                case P_VAL:
                    spread(*p.lv, [&](int at, int e) { D[p.off + at] = e < 0 ? 0.0 : p.lv->val[e]; });
                    break;
                case P_VAL32:
                    spread(*p.lv, [&](int at, int e) {
                        F[p.off + at] = e < 0 ? 0.0f : static_cast<float>(p.lv->val[e]);
                    });
                    break;
                case P_PTR: case P_AGG: case P_CPTR: case P_CIDX: {
                    const auto &v = *static_cast<const std::vector<int> *>(p.src);
                    std::copy(v.begin(), v.end(), I.get() + p.off);
                    std::fill(I.get() + p.off + v.size(), I.get() + p.off + (v.size() + 7) / 8 * 8, 0);
                    break;
                }
                case P_RDG: case P_INV: {
                    const auto &v = *static_cast<const std::vector<double> *>(p.src);
                    std::copy(v.begin(), v.end(), D.get() + p.off);
                    std::fill(D.get() + p.off + v.size(), D.get() + p.off + (v.size() + 3) / 4 * 4, 0.0);
                    break;
                }
                default: {
                    const auto &v = *static_cast<const std::vector<double> *>(p.src);
                    for (size_t e = 0; e < v.size(); ++e)
                        F[p.off + e] = static_cast<float>(v[e]);
                    std::fill(F.get() + p.off + v.size(), F.get() + p.off + (v.size() + 7) / 8 * 8, 0.0f);
                }
                }
            }
            for (int s = nextRhs++; s < n; s = nextRhs++)
                std::memcpy(hb.get() + L.xOff[s], systems[s].source, sizeof(double) * L.rows[s]);
        };
        std::vector<std::thread> pool;
        for (int t = 1; t < nt; ++t)
            pool.emplace_back(work);
        work();
        for (auto &t : pool)
            t.join();
    }
    L.dI.ensure(std::max<size_t>(nI, 1) * sizeof(int32_t));
    L.dD.ensure(std::max<size_t>(nD, 1) * sizeof(double));
    L.dF.ensure(std::max<size_t>(nF, 1) * sizeof(float));
    check(cudaMemcpy(L.dI.p, I.get(), nI * sizeof(int32_t), cudaMemcpyHostToDevice), "upload");
    check(cudaMemcpy(L.dD.p, D.get(), nD * sizeof(double), cudaMemcpyHostToDevice), "upload");
    if (nF)
        check(cudaMemcpy(L.dF.p, F.get(), nF * sizeof(float), cudaMemcpyHostToDevice), "upload");
    for (const Piece &p : pieces) {
        rq::DevLinSys &d = byIndex[p.s];
        rq::DevLinLevel &dl = d.lev[p.l];
        const int32_t *ip = L.dI.as<int32_t>() + p.off;
        const double *dp = L.dD.as<double>() + p.off;
        const float *fp = L.dF.as<float>() + p.off;
        switch (p.what) {
        case P_PTR: dl.ptr = ip; break;
        case P_COL: dl.col = ip; break;
        case P_VAL: dl.val = dp; break;
        case P_RDG: dl.rdg = dp; break;
        case P_VAL32: dl.val32 = fp; break;
        case P_RDG32: dl.rdg32 = fp; break;
        case P_AGG: dl.agg = ip; break;
        case P_CPTR: dl.childPtr = ip; break;
        case P_CIDX: dl.childIdx = ip; break;
        case P_INV: d.inv = dp; break;
        case P_INV32: d.inv32 = fp; break;
        }
    }
    // right-hand sides (gathered above), solutions and results
    L.dB.ensure(sizeof(double) * L.totalRows);
    L.dX.ensure(sizeof(double) * L.totalRows);
    L.dOut.ensure(sizeof(rq::LinOut) * n);
    check(cudaMemcpy(L.dB.p, hb.get(), sizeof(double) * L.totalRows, cudaMemcpyHostToDevice), "rhs");
    for (int s = 0; s < n; ++s) {
        byIndex[s].b = L.dB.as<double>() + L.xOff[s];
        byIndex[s].x = L.dX.as<double>() + L.xOff[s];
        byIndex[s].out = L.dOut.as<rq::LinOut>() + s;
    }
    // queue order: by launch shape, largest systems first (longest-processing-time)
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return L.rows[a] > L.rows[b]; });
    L.sys.clear();
    long wsTotal = 0;
    std::vector<int> queue(n);
    for (int k = 0; k < n; ++k)
        queue[k] = L.rows[order[k]];
    const size_t localMost = *std::max_element(localOf.begin(), localOf.end());
    const int halvings =
        linHalvings(queue, [&](int threads, int c) {
            return rq::linConcurrent({threads, c, localMost});
        });
    for (int s : order) {
        byIndex[s].slices = linSlices(L.rows[s]);
        const int threads = linThreads(L.rows[s]);
        const int cluster = std::max(1, byIndex[s].slices >> halvings);
        if (L.groups.empty() || L.groups.back().shape.cluster != cluster ||
            L.groups.back().shape.threads != threads) {
            L.groups.emplace_back();
            L.groups.back().first = static_cast<int>(L.sys.size());
            L.groups.back().shape = {threads, cluster, 0};
        }
        rq_linsys::Group &g = L.groups.back();
        ++g.count;
        g.wsStride = std::max(g.wsStride, wsOf[s]);
        g.shape.localBytes = std::max(g.shape.localBytes, localOf[s]);
        L.sys.push_back(byIndex[s]);
    }
    for (size_t k = 0; k < L.groups.size(); ++k) {
        rq_linsys::Group &g = L.groups[k];
        const int atOnce = rq::linConcurrent(g.shape);
        if (atOnce < 1)
            throw RqError(RQ_E_CUDA, "linear solve kernel does not fit on an SM");
        g.slots = std::min(g.count, atOnce);
        g.wsOff = wsTotal;
        wsTotal += g.wsStride * g.slots;
        if (k > 0) {
            check(cudaStreamCreateWithFlags(&g.stream, cudaStreamNonBlocking), "stream");
            check(cudaEventCreateWithFlags(&g.done, cudaEventDisableTiming), "event");
        }
    }
    if (L.groups.size() > 1)
        check(cudaEventCreateWithFlags(&L.fork, cudaEventDisableTiming), "event");
    L.dWs.ensure(sizeof(double) * wsTotal);
    L.dSys.ensure(sizeof(rq::DevLinSys) * n);
    L.dNext.ensure(sizeof(int) * L.groups.size());
}

// One launch per shape, side by side: the first on the caller's stream, the others
// on streams of the handle that fork from it and join it.
void launchLinsys(rq_linsys &L, int maxIter, double tol, cudaStream_t stream) {
    for (auto &d : L.sys) {
        d.maxIter = maxIter;
        d.tol = tol;
    }
    check(cudaMemcpyAsync(L.dSys.p, L.sys.data(), sizeof(rq::DevLinSys) * L.nsys,
                          cudaMemcpyHostToDevice, stream), "systems");
    check(cudaMemsetAsync(L.dNext.p, 0, sizeof(int) * L.groups.size(), stream), "counter");
    if (L.fork)
        check(cudaEventRecord(L.fork, stream), "event record");
    for (size_t k = 0; k < L.groups.size(); ++k) {
        const rq_linsys::Group &g = L.groups[k];
        const cudaStream_t st = k ? g.stream : stream;
        if (k)
            check(cudaStreamWaitEvent(st, L.fork, 0), "stream wait");
        check(rq::launchLinear(L.dSys.as<rq::DevLinSys>() + g.first, g.count,
                               L.dNext.as<int>() + k, L.dWs.as<double>() + g.wsOff, g.wsStride,
                               g.slots, g.shape, st), "linear solve launch");
        if (k) {
            check(cudaEventRecord(g.done, st), "event record");
            check(cudaStreamWaitEvent(stream, g.done, 0), "stream wait");
        }
    }
}

void fetchLinsys(rq_linsys &L, double *const *x, rq_solver_result *results) {
    static_assert(sizeof(rq::LinOut) == sizeof(rq_solver_result), "result layout");
    if (results)
        check(cudaMemcpy(results, L.dOut.p, sizeof(rq::LinOut) * L.nsys, cudaMemcpyDeviceToHost),
              "results");
    // Large solutions go straight into the caller's arrays, runs of small ones through one
    // buffer: a copy of its own costs each system about 13 us, as long as the second copy of
    // 12000 rows (256 systems of 24 x 24: a solve of 4.2 ms each by itself, 1.4 in one buffer).
    constexpr int kLarge = 12288;
    constexpr int64_t kRun = 1 << 20;
    std::vector<double> buffer;
    for (int s = 0, end; x && s < L.nsys; s = end) {
        const double *from = L.dX.as<double>() + L.xOff[s];
        int64_t cnt = L.rows[s];
        end = s + 1;
        while (L.rows[s] < kLarge && end < L.nsys && L.rows[end] < kLarge && cnt + L.rows[end] <= kRun)
            cnt += L.rows[end++];
        if (end == s + 1) {
            check(cudaMemcpy(x[s], from, sizeof(double) * cnt, cudaMemcpyDeviceToHost), "x");
            continue;
        }
        buffer.resize(std::max<size_t>(buffer.size(), cnt));
        check(cudaMemcpy(buffer.data(), from, sizeof(double) * cnt, cudaMemcpyDeviceToHost), "x");
        for (int k = s; k < end; ++k)
            std::memcpy(x[k], buffer.data() + (L.xOff[k] - L.xOff[s]), sizeof(double) * L.rows[k]);
    }
}

} // namespace

extern "C" {
int rq_linsys_create(const rq_ldu *systems, int32_t n_systems, int32_t kind, int32_t precision,
                     rq_linsys **out) {
    return guarded([&] {
        if (!systems || n_systems < 1 || !out)
            throw std::invalid_argument("null argument");
        *out = nullptr;
        if (kind == 3)
            throw RqError(RQ_E_UNSUPPORTED, "the Gauss-Seidel solver is not on the GPU path");
        if (kind < 0 || kind > 2)
            throw std::invalid_argument("unknown linear solver kind");
        if (precision != RQ_PREC_FP64 && precision != RQ_PREC_MIXED)
            throw std::invalid_argument("unknown precision");
        auto L = std::make_unique<rq_linsys>();
        buildLinsys(*L, systems, n_systems, kind, precision);
        *out = L.release();
    });
}

int rq_linsys_solve(rq_linsys *L, int32_t max_iter, double tol, double *const *x,
                    rq_solver_result *results) {
    return guarded([&] {
        if (!L)
            throw std::invalid_argument("null argument");
        std::lock_guard<std::mutex> lock(L->mu);
        checkSolveArgs(max_iter, tol);
        if (x)
            for (int s = 0; s < L->nsys; ++s) {
                if (!x[s])
                    throw std::invalid_argument("null initial guess");
                for (int i = 0; i < L->rows[s]; ++i)
                    if (!std::isfinite(x[s][i]))
                        throw std::invalid_argument("linear solve initial values must be finite");
            }
        if (x) {
            std::vector<double> hx(L->totalRows);
            for (int s = 0; s < L->nsys; ++s)
                std::memcpy(hx.data() + L->xOff[s], x[s], sizeof(double) * L->rows[s]);
            check(cudaMemcpy(L->dX.p, hx.data(), sizeof(double) * hx.size(), cudaMemcpyHostToDevice), "x");
        } else {
            check(cudaMemset(L->dX.p, 0, sizeof(double) * L->totalRows), "x");
        }
        launchLinsys(*L, max_iter, tol, nullptr);
        check(cudaStreamSynchronize(nullptr), "linear solve");
        fetchLinsys(*L, x, results);
    });
}

int rq_linsys_solve_device(rq_linsys *L, int32_t max_iter, double tol, void *stream) {
    return guarded([&] {
        if (!L)
            throw std::invalid_argument("null argument");
        std::lock_guard<std::mutex> lock(L->mu);
        checkSolveArgs(max_iter, tol);
        const cudaStream_t st = static_cast<cudaStream_t>(stream);
        check(cudaMemsetAsync(L->dX.p, 0, sizeof(double) * L->totalRows, st), "x");
        launchLinsys(*L, max_iter, tol, st);
    });
}

int rq_linsys_results(rq_linsys *L, rq_solver_result *results, double *const *x) {
    return guarded([&] {
        if (!L)
            throw std::invalid_argument("null argument");
        std::lock_guard<std::mutex> lock(L->mu);
        check(cudaDeviceSynchronize(), "linear solve");
        fetchLinsys(*L, x, results);
    });
}

int rq_linsys_info(const rq_linsys *L, int32_t *n_systems, int64_t *total_rows, int64_t *total_nnz,
                   int32_t *max_levels) {
    return guarded([&] {
        if (!L)
            throw std::invalid_argument("null argument");
        if (n_systems)
            *n_systems = L->nsys;
        if (total_rows)
            *total_rows = L->totalRows;
        if (total_nnz)
            *total_nnz = L->totalNnz;
        if (max_levels)
            *max_levels = L->maxLevels;
    });
}

int rq_linsys_destroy(rq_linsys *L) {
    return guarded([&] { delete L; });
}

int rq_linear_solve_batch(const rq_ldu *systems, int32_t n_systems, double *const *x,
                          int32_t max_iter, double tol, int32_t kind, int32_t precision,
                          rq_solver_result *results) {
    rq_linsys *L = nullptr;
    int rc = rq_linsys_create(systems, n_systems, kind, precision, &L);
    if (rc != RQ_OK)
        return rc;
    rc = rq_linsys_solve(L, max_iter, tol, x, results);
    rq_linsys_destroy(L);
    return rc;
}

int rq_linear_solve(const rq_ldu *A, double *x, int32_t max_iter, double tol, int32_t kind,
                    rq_solver_result *result) {
    if (!x) {
        g_error = "null argument";
        return RQ_E_INVALID;
    }
    double *xs[1] = {x};
    return rq_linear_solve_batch(A, 1, xs, max_iter, tol, kind, RQ_PREC_FP64, result);
}

} // extern "C"
