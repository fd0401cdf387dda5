// solveCG / solveBiCGStab on a caller's CSR matrix (src/common/src/Matrix.cpp:153-319):
// the drop-in for the reference's linear-solver call surface.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "ctx.h"
#include "solvers.cuh"
#include "persist.cuh"

namespace cfg
{

namespace
{

struct DevBuf
{
    std::vector<void*> ptrs;
    cudaStream_t s;
    template <class T>
    T* get(size_t n)
    {
        void* p = nullptr;
        CFG_CUDA(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
        ptrs.push_back(p);
        CFG_CUDA(cudaMemsetAsync(p, 0, std::max<size_t>(n, 1) * sizeof(T), s));
        return static_cast<T*>(p);
    }
    ~DevBuf()
    {
        cudaStreamSynchronize(s);
        for (void* p : ptrs) cudaFree(p);
    }
};

__global__ void k_diag_from_sell(DMat A, const int* __restrict__ isDiag, const double* __restrict__ val, double* d)
{
    ROW_LOOP(c, A.n)
    {
        const int sl = c >> 5, lane = c & 31;
        double v = 0.0;
        for (int e = A.start[sl] + lane; e < A.start[sl + 1]; e += 32)
        {
            if (A.col[e] < 0) break;
            if (isDiag[e])
            {
                v = val[e];
                break;
            }
        }
        d[c] = v;
    }
}

/// The solve as one resident kernel that reads the caller's CSR as it is:
/// one allocation, the arrays copied in, the kernel, the solution copied out.
/// False when the system does not fit (a row of more than kResW entries, more
/// rows than a team holds).  A 30,044-row BiCGStab call took 9.4 ms with the
/// SELL conversion on the host, an allocation per vector and four launches
/// per iteration.
bool residentSolve(int device, int n, int maxRow, const int64_t* rs, const int64_t* cols, const double* vals,
                   const double* b, double* x, double tol, int maxIter, int method, cfg_solver_report* rep)
{
    int sms = 0, coop = 0;
    CFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    CFG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    const TeamPlan tp = maxRow <= kResW ? teamPlanOf(n, 1, largestCluster(device), sms, coop != 0) : TeamPlan{};
    if (!tp.blocks) return false;
    const size_t N = static_cast<size_t>(n), nnz = static_cast<size_t>(rs[n]);
    size_t bytes = 0;
    auto place = [&](size_t size) {
        const size_t at = bytes;
        bytes += (size + 255) / 256 * 256;
        return at;
    };
    // the zeroed part first: counters, the state and the failure flag
    struct Outcome
    {
        SolveState st;
        int failed;
    };
    const size_t oCount = place(kTeamsMax * kCountStride * sizeof(unsigned)), oOutcome = place(sizeof(Outcome)),
                 zeroed = bytes;
    const size_t oRs = place((N + 1) * sizeof(int64_t)), oCols = place(nnz * sizeof(int64_t)),
                 oVals = place(nnz * sizeof(double)), oB = place(N * sizeof(double)), oX = place(N * sizeof(double)),
                 oG = place(N * sizeof(double)), oPart = place(teamPartSize(n) * sizeof(double));
    cudaStream_t s;
    CFG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct Guard
    {
        cudaStream_t s;
        unsigned char* p = nullptr;
        ~Guard()
        {
            cudaStreamSynchronize(s);
            cudaFree(p);
            cudaStreamDestroy(s);
        }
    } g{s};
    CFG_CUDA(cudaMalloc(&g.p, bytes));
    unsigned char* d = g.p;
    auto in = [&](size_t at, const void* src, size_t size) {
        if (size) CFG_CUDA(cudaMemcpyAsync(d + at, src, size, cudaMemcpyHostToDevice, s));
    };
    CFG_CUDA(cudaMemsetAsync(d, 0, zeroed, s));
    in(oRs, rs, (N + 1) * sizeof(int64_t));
    in(oCols, cols, nnz * sizeof(int64_t));
    in(oVals, vals, nnz * sizeof(double));
    in(oB, b, N * sizeof(double));
    in(oX, x, N * sizeof(double));
    using View = CsrView<long long>;
    static_assert(sizeof(long long) == sizeof(int64_t), "64-bit indices");
    const View A{n, reinterpret_cast<const long long*>(d + oRs), reinterpret_cast<const long long*>(d + oCols),
                 reinterpret_cast<const double*>(d + oVals)};
    double* const db = reinterpret_cast<double*>(d + oB);
    double* const dx = reinterpret_cast<double*>(d + oX);
    double* const dg = reinterpret_cast<double*>(d + oG);
    Outcome* const out = reinterpret_cast<Outcome*>(d + oOutcome);
    const PersArgs t{tol, maxIter, 0, tp.chunk, &out->st, nullptr,
                     teamMem(tp, n, reinterpret_cast<unsigned*>(d + oCount), reinterpret_cast<double*>(d + oPart),
                             &out->failed)};
    dispatchK<kRes1K>(tp.K, [&](auto Kc) {
        constexpr int K = decltype(Kc)::value;
        if (method == CFG_SOLVE_CG)
        {
            const PersCg<View> a{A, db, dx, dg, nullptr, nullptr, 0};
            const size_t smem = resident_smem(K, 1, true);
            if (tp.cluster) launchTeam(tp, 1, k_pers_cg<K, ClusterTeam, false, View>, a, t, smem, s);
            else launchTeam(tp, 1, k_pers_cg<K, GridTeam, false, View>, a, t, smem, s);
        }
        else
        {
            const PersBi<View> a{A, V3P{{db, db, db}}, V3P{{dx, dx, dx}}, V3P{{dg, dg, dg}}};
            const size_t smem = resident_smem(K, 1, false);
            if (tp.cluster) launchTeam(tp, 1, k_pers_bicg<K, ClusterTeam, 1, View>, a, t, smem, s);
            else launchTeam(tp, 1, k_pers_bicg<K, GridTeam, 1, View>, a, t, smem, s);
        }
    });
    // the caller's x changes only once the solve is known to have ended well
    Outcome got;
    CFG_CUDA(cudaMemcpyAsync(&got, out, sizeof got, cudaMemcpyDeviceToHost, s));
    CFG_CUDA(cudaStreamSynchronize(s));
    if (got.failed) fail(CFG_ECUDA, "sparse solve: a wait inside a kernel ran out");
    CFG_CUDA(cudaMemcpyAsync(x, dx, N * sizeof(double), cudaMemcpyDeviceToHost, s));
    CFG_CUDA(cudaStreamSynchronize(s));
    const SolveState& h = got.st;
    rep->iterations = h.it[0];
    rep->converged = h.conv[0];
    rep->initial_residual = h.init[0];
    rep->final_residual = (h.conv[0] && h.it[0] == 0) ? h.init[0] : h.fin[0];
    return true;
}

}  // namespace

void Ctx::sparseSolve(int device, int64_t n64, const int64_t* rs, const int64_t* cols, const double* vals,
                      const double* b, double* x, double tol, int maxIter, int method, cfg_solver_report* rep)
{
    if (n64 <= 0 || n64 >= (1LL << 30)) fail(CFG_EINVAL, "sparse solve: matrix size out of range");
    const int n = static_cast<int>(n64);
    int maxRow = 0;
    for (int r = 0; r < n; ++r)
    {
        maxRow = std::max<int>(maxRow, static_cast<int>(std::min<int64_t>(rs[r + 1] - rs[r], 1 << 30)));
        if (rs[r + 1] < rs[r]) fail(CFG_EINVAL, "sparse solve: row offsets not ascending");
        for (int64_t k = rs[r]; k < rs[r + 1]; ++k)
            if (cols[k] < 0 || cols[k] >= n) fail(CFG_EINVAL, "sparse solve: column out of range");
    }
    CFG_CUDA(cudaSetDevice(device));
    const SolveScope scope(device);
    if (rs[0] == 0 && residentSolve(device, n, maxRow, rs, cols, vals, b, x, tol, maxIter, method, rep)) return;
    cudaStream_t s;
    CFG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamGuard
    {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } sg{s};
    DevBuf buf;
    buf.s = s;
    // SELL-32 with each row's entries in the caller's order
    const int nS = (n + 31) / 32;
    std::vector<int> start(nS + 1, 0);
    for (int sl = 0; sl < nS; ++sl)
    {
        int w = 0;
        for (int l = 0; l < 32 && 32 * sl + l < n; ++l) w = std::max<int>(w, static_cast<int>(rs[32 * sl + l + 1] - rs[32 * sl + l]));
        start[sl + 1] = start[sl] + 32 * w;
    }
    std::vector<int> col(start[nS], -1), isDiag(start[nS], 0);
    std::vector<double> val(start[nS], 0.0);
    std::vector<char> seenDiag(n, 0);
    for (int r = 0; r < n; ++r)
    {
        const int sl = r >> 5, l = r & 31;
        for (int64_t k = rs[r]; k < rs[r + 1]; ++k)
        {
            const int e = start[sl] + 32 * static_cast<int>(k - rs[r]) + l;
            col[e] = static_cast<int>(cols[k]);
            val[e] = vals[k];
            // SparseMatrix::diagonal takes the first entry in the diagonal column
            if (cols[k] == r && !seenDiag[r])
            {
                isDiag[e] = 1;
                seenDiag[r] = 1;
            }
        }
    }
    int sms = 0;
    CFG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const int G = std::max(1, std::min((n + TPB - 1) / TPB, sms * 8));
    const int GS = std::max(1, (n + RPT * TPB - 1) / (RPT * TPB));
    int maxW = 0;
    for (int sl = 0; sl < nS; ++sl) maxW = std::max(maxW, (start[sl + 1] - start[sl]) / 32);
    int* dStart = buf.get<int>(start.size());
    int* dCol = buf.get<int>(col.size());
    int* dIsDiag = buf.get<int>(isDiag.size());
    double* dVal = buf.get<double>(val.size());
    double* dDiag = buf.get<double>(n);
    double* db = buf.get<double>(n);
    double* dx = buf.get<double>(n);
    CFG_CUDA(cudaMemcpyAsync(dStart, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    CFG_CUDA(cudaMemcpyAsync(dCol, col.data(), col.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    CFG_CUDA(cudaMemcpyAsync(dIsDiag, isDiag.data(), isDiag.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    CFG_CUDA(cudaMemcpyAsync(dVal, val.data(), val.size() * sizeof(double), cudaMemcpyHostToDevice, s));
    CFG_CUDA(cudaMemcpyAsync(db, b, n * sizeof(double), cudaMemcpyHostToDevice, s));
    CFG_CUDA(cudaMemcpyAsync(dx, x, n * sizeof(double), cudaMemcpyHostToDevice, s));
    const DMat A{n, dStart, dCol};
    k_diag_from_sell<<<G, TPB, 0, s>>>(A, dIsDiag, dVal, dDiag);
    double* partials = buf.get<double>(16 * static_cast<size_t>(std::max(G, GS)));
    SolveState* st = buf.get<SolveState>(1);
    SolveState* hst = nullptr;
    CFG_CUDA(cudaMallocHost(&hst, sizeof(SolveState)));
    struct HostGuard
    {
        SolveState* p;
        ~HostGuard() { cudaFreeHost(p); }
    } hg{hst};
    SolveState init{};
    init.tol = tol;
    init.maxIter = maxIter;
    init.nComp = 1;
    CFG_CUDA(cudaMemcpyAsync(st, &init, sizeof(SolveState), cudaMemcpyHostToDevice, s));
    auto poll = [&]() {
        CFG_CUDA(cudaMemcpyAsync(hst, st, sizeof(SolveState), cudaMemcpyDeviceToHost, s));
        CFG_CUDA(cudaStreamSynchronize(s));
        return hst->allDone != 0;
    };
    auto run = [&](auto Wc) {
        constexpr int W = decltype(Wc)::value;
        if (method == CFG_SOLVE_CG)
        {
            double* r = buf.get<double>(n);
            double* p = buf.get<double>(n);
            double* Ap = buf.get<double>(n);
            k_cg_init<W><<<GS, TPB, 0, s>>>(A, dVal, dDiag, db, dx, r, p, partials, st);
            CFG_CUDA(cudaGetLastError());
            for (int launched = 0, chunk = 8; !poll() && launched < maxIter; chunk = std::min(2 * chunk, 64))
            {
                const int m = std::min(chunk, maxIter - launched);
                for (int k = 0; k < m; ++k)
                {
                    k_cg_spmv<W><<<GS, TPB, 0, s>>>(A, dVal, p, Ap, partials, st);
                    k_cg_update<double><<<GS, TPB, 0, s>>>(n, dDiag, p, Ap, dx, r, partials, st);
                    k_cg_p<double><<<GS, TPB, 0, s>>>(n, dDiag, r, p, st);
                }
                CFG_CUDA(cudaGetLastError());
                launched += m;
            }
        }
        else
        {
            V3P r{}, r0{}, p{}, v{}, t{}, z{}, bb{}, xx{};
            for (int q = 0; q < 3; ++q)
            {
                r.c[q] = buf.get<double>(n);
                r0.c[q] = buf.get<double>(n);
                p.c[q] = buf.get<double>(n);
                v.c[q] = buf.get<double>(n);
                t.c[q] = buf.get<double>(n);
                z.c[q] = buf.get<double>(n);
                bb.c[q] = db;
                xx.c[q] = dx;
            }
            double* invD = buf.get<double>(n);
            k_bi_init<W, 1><<<GS, TPB, 0, s>>>(A, dVal, dDiag, invD, bb, xx, r, r0, p, v, partials, st);
            CFG_CUDA(cudaGetLastError());
            for (int launched = 0, chunk = 4; !poll() && launched < maxIter; chunk = std::min(2 * chunk, 32))
            {
                const int m = std::min(chunk, maxIter - launched);
                for (int k = 0; k < m; ++k)
                {
                    k_bi_p<1><<<GS, TPB, 0, s>>>(n, invD, r, p, v, z, st);
                    k_bi_spmv1<W, 1><<<GS, TPB, 0, s>>>(A, dVal, z, v, r0, partials, st);
                    k_bi_spmv2<W, 1><<<GS, TPB, 0, s>>>(A, dVal, invD, r, v, t, partials, st);
                    k_bi_x<1><<<GS, TPB, 0, s>>>(n, invD, xx, z, v, t, r, r0, partials, st);
                }
                CFG_CUDA(cudaGetLastError());
                launched += m;
            }
        }
    };
    if (maxW <= 7) run(std::integral_constant<int, 7>{});
    else if (maxW <= 16) run(std::integral_constant<int, 16>{});
    else run(std::integral_constant<int, 0>{});
    CFG_CUDA(cudaMemcpyAsync(x, dx, n * sizeof(double), cudaMemcpyDeviceToHost, s));
    CFG_CUDA(cudaStreamSynchronize(s));
    rep->iterations = hst->it[0];
    rep->converged = hst->conv[0];
    rep->initial_residual = hst->init[0];
    rep->final_residual = (hst->conv[0] && hst->it[0] == 0) ? hst->init[0] : hst->fin[0];
}

}  // namespace cfg
