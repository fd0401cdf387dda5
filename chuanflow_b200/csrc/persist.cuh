// The Krylov solves as one kernel each, with the system resident on the chip:
// CG (Jacobi or multicolour DIC) and the Jacobi BiCGStab of solvers.cuh /
// dic.cuh, every iteration inside a team of blocks (team.cuh).  A block keeps
// its rows' matrix entries and the vector its neighbours gather in shared
// memory and every other vector in registers; an iteration touches global
// memory only for values a grid team's blocks read from each other.  The
// arithmetic of each vector element is that of the per-iteration kernels, and
// so is the order of the reductions when those run one row per thread.
#pragma once

#include "dic.cuh"
#include "team.cuh"

namespace cfg
{

/// entries per row the resident kernels hold: hexahedra (6 neighbours and
/// the diagonal), tetrahedra and prisms fit
constexpr int kResW = 7;

/// The matrix of a resident solve: row c's entries in order, e = first(c),
/// first(c) + step, ... while live(e, c); its diagonal as the solvers take it.
struct SellView
{
    DMat A;
    const double* val;
    const double* diag_;
    static constexpr int step = 32;
    static constexpr bool checked = false;  // every row is known to fit kResW
    __device__ __forceinline__ int n() const { return A.n; }
    __device__ __forceinline__ long long first(int c) const { return __ldg(A.start + (c >> 5)) + (c & 31); }
    __device__ __forceinline__ long long end(int c) const { return __ldg(A.start + (c >> 5) + 1); }
    __device__ __forceinline__ int col(long long e) const { return __ldg(A.col + e); }
    __device__ __forceinline__ double value(long long e) const { return __ldg(val + e); }
    __device__ __forceinline__ double diag(int c) const { return __ldg(diag_ + c); }
};
/// A caller's CSR with 32- or 64-bit indices, as it is.
template <class I>
struct CsrView
{
    int rows;
    const I *rs, *cols;
    const double* val;
    static constexpr int step = 1;
    static constexpr bool checked = true;
    __device__ __forceinline__ int n() const { return rows; }
    __device__ __forceinline__ long long first(int c) const { return __ldg(rs + c); }
    __device__ __forceinline__ long long end(int c) const { return __ldg(rs + c + 1); }
    __device__ __forceinline__ int col(long long e) const { return static_cast<int>(__ldg(cols + e)); }
    __device__ __forceinline__ double value(long long e) const { return __ldg(val + e); }
    /// the first entry in the diagonal column, else 0 (SparseMatrix::diagonal)
    __device__ __forceinline__ double diag(int c) const
    {
        for (long long e = first(c); e < end(c); ++e)
            if (col(e) == c) return value(e);
        return 0.0;
    }
};

/// A solve's arguments beyond its vectors: the stopping test, the rows per
/// block (contiguous), where the outcome goes, the optional {iterations,
/// unconverged} sums of an outer iteration, and for a matrix whose rows no host
/// has measured a zero word that is set, with nothing else written, when one
/// has more than kResW entries.
struct PersArgs
{
    double tol;
    int maxIter;
    int normType;
    int chunk;
    SolveState* st;
    double* tally;
    TeamMem g;
    int* wide = nullptr;
};

/// whether the team leaves: a row is too long, or a wait ran out (asked first:
/// then another block may still be writing the word)
template <class Team, class Mat>
__device__ __forceinline__ bool too_wide(Team& tm, const Mat& A, int lo, int cnt, int* wide)
{
    bool mine = false;
    for (int i = threadIdx.x; i < cnt; i += kTeamThreads) mine |= A.end(lo + i) - A.first(lo + i) > kResW;
    volatile int* const w = wide;
    if (__syncthreads_or(mine) && threadIdx.x == 0) *w = 1;
    tm.sync();
    return tm.dead() || *w != 0;
}

/// whether a solve keeps its matrix entries in registers
__host__ __device__ constexpr bool resident_regs(int K, int NC, bool jacobiCg) { return NC == 1 && (K == 1 || (K == 2 && jacobiCg)); }
/// whether the three-component BiCGStab keeps x in shared memory (two rows
/// per thread do not leave it registers)
__host__ __device__ constexpr bool resident_xs(int K, int NC) { return NC == 3 && K > 1; }

/// a component's part of the gather vector: its slots, then a slot that holds
/// zero for the entries a row does not have (a real slot's infinity or NaN
/// would reach rows that are not coupled to it), padded to 16 bytes
__host__ __device__ constexpr int resident_stride(int K) { return K * kTeamThreads + 2; }

/// dynamic shared memory of a block holding K * kTeamThreads rows of an
/// NC-component solve: gather vector, values and column codes, x
__host__ __device__ constexpr size_t resident_smem(int K, int NC, bool jacobiCg)
{
    return static_cast<size_t>(NC) * resident_stride(K) * sizeof(double) +
           static_cast<size_t>(K) * kTeamThreads *
           ((resident_regs(K, NC, jacobiCg) ? 0 : kResW * (sizeof(double) + sizeof(int))) +
            (resident_xs(K, NC) ? NC * sizeof(double) : 0));
}

/// A block's rows of the matrix and the vector the neighbours gather.
/// Row slot i of the block is row lo + i; thread t owns slots t + k T.
/// A column code is the slot of a row of this block, or the complement of
/// where another block keeps it: its shared::cluster address (cluster
/// team), its row in the team's global copy of the vector (grid team).
template <int K, int NC, class Team, bool kRegs>
struct Resident
{
    static constexpr int S = K * kTeamThreads, BS = resident_stride(K);
    static constexpr bool kCluster = Team::kCluster;
    // kRegs: the entries are in registers (one component, few rows per
    // thread), and a row's product reads shared memory for the gathered
    // values only (8 of 20 bytes per entry)
    double rv[kRegs ? K : 1][kResW];
    int rc[kRegs ? K : 1][kResW];
    double* val;  // [kResW][S]
    double* buf;  // [NC][BS]
    int* code;    // [kResW][S]
    V3P shared;   // the grid team's copy of buf
    int lo, cnt;

    __device__ Resident(unsigned char* smem, V3P g, int lo_, int cnt_) : shared(g), lo(lo_), cnt(cnt_)
    {
        buf = reinterpret_cast<double*>(smem);
        val = buf + NC * BS;
        code = reinterpret_cast<int*>(val + (kRegs ? 0 : kResW * S));
        if (threadIdx.x < NC) buf[threadIdx.x * BS + S] = 0.0;
    }
    /// the block's entries; slots past the last row and past a row's last entry
    /// are zero values at the zero slot
    template <class Mat>
    __device__ __forceinline__ void load(const Mat& A, int chunk, int rank)
    {
        const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(buf));
#pragma unroll
        for (int s = 0; s < K; ++s)
        {
            const int i = threadIdx.x + s * kTeamThreads, c = lo + i;
            long long e0 = 0, e1 = 0;
            if (i < cnt)
            {
                e0 = A.first(c);
                e1 = A.end(c);
            }
#pragma unroll
            for (int k = 0; k < kResW; ++k)
            {
                const long long e = e0 + Mat::step * k;
                const int col = e < e1 ? A.col(e) : -1;
                int cd = S;
                if (col >= 0)
                {
                    const int owner = col / chunk, slot = col - owner * chunk;
                    if (owner == rank) cd = slot;
                    else if constexpr (kCluster)
                    {
                        unsigned remote;
                        asm("mapa.shared::cluster.u32 %0, %1, %2;"
                            : "=r"(remote)
                            : "r"(base + 8u * static_cast<unsigned>(slot)), "r"(owner));
                        cd = ~static_cast<int>(remote);
                    }
                    else cd = ~col;
                }
                const double ve = col >= 0 ? A.value(e) : 0.0;
                if constexpr (kRegs)
                {
                    rv[s][k] = ve;
                    rc[s][k] = cd;
                }
                else
                {
                    val[k * S + i] = ve;
                    code[k * S + i] = cd;
                }
            }
        }
    }
    __device__ __forceinline__ double gather(int cd, int q) const
    {
        if (cd >= 0) return buf[q * BS + cd];
        if constexpr (kCluster)
        {
            double v;
            asm volatile("ld.shared::cluster.f64 %0, [%1];"
                         : "=d"(v)
                         : "r"(static_cast<unsigned>(~cd) + 8u * static_cast<unsigned>(q * BS)));
            return v;
        }
        else return __ldcg(shared.c[q] + ~cd);
    }
    __device__ __forceinline__ double value(int s, int k) const
    {
        if constexpr (kRegs) return rv[s][k];
        else return val[k * S + threadIdx.x + s * kTeamThreads];
    }
    __device__ __forceinline__ int codeOf(int s, int k) const
    {
        if constexpr (kRegs) return rc[s][k];
        else return code[k * S + threadIdx.x + s * kTeamThreads];
    }
    /// y = row s of this thread times the gather vector, entries in row order
    __device__ __forceinline__ void row(int s, double (&y)[NC]) const
    {
        double x[kResW][NC], v[kResW];
#pragma unroll
        for (int k = 0; k < kResW; ++k)
        {
            const int cd = codeOf(s, k);
            v[k] = value(s, k);
#pragma unroll
            for (int q = 0; q < NC; ++q) x[k][q] = gather(cd, q);
        }
#pragma unroll
        for (int q = 0; q < NC; ++q)
        {
            y[q] = 0.0;
#pragma unroll
            for (int k = 0; k < kResW; ++k) y[q] += v[k] * x[k][q];
        }
    }
    /// the same over the entries whose bit is set in `mask`
    __device__ __forceinline__ double masked(int s, unsigned mask) const
    {
        double y = 0.0, x[kResW];
#pragma unroll
        for (int k = 0; k < kResW; ++k) x[k] = (mask >> k & 1u) ? gather(codeOf(s, k), 0) : 0.0;
#pragma unroll
        for (int k = 0; k < kResW; ++k)
            if (mask >> k & 1u) y += value(s, k) * x[k];
        return y;
    }
    /// the gather vector's value of slot i, for this block and the others
    __device__ __forceinline__ void put(int i, int q, double v)
    {
        buf[q * BS + i] = v;
        if constexpr (!kCluster)
            if (i < cnt) shared.c[q][lo + i] = v;
    }
};

template <class Mat>
struct PersCg
{
    Mat A;
    const double* b;
    double* x;
    double* g;  // a grid team's copy of the gather vector
    // DIC: 1/rD per row, colours, each row's colour
    const double* rDinv;
    const int* colour;
    int nColours;
};

/// z = M^-1 r of the multicolour DIC (k_dic_fwd, k_dic_bwd) and this
/// thread's r z: one team barrier between colours, z passed to the
/// neighbours through the gather vector.  On entry z = rDinv r is there
/// already (the first colour has no lower entries), put before the last
/// reduction, whose barrier made it visible.
template <int K, class Team, class Res>
__device__ __forceinline__ void pers_dic(Team& tm, Res& R, int C, const double (&r)[K], const double (&rd)[K],
                                           const int (&col)[K], const unsigned (&lower)[K], const unsigned (&upper)[K],
                                         double (&z)[K], double (&rz)[K][1])
{
    for (int c = 1; c < C; ++c)
    {
        if (c > 1)
        {
            tm.sync();
            if (tm.dead()) return;
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (col[k] != c) continue;
            const int i = threadIdx.x + k * kTeamThreads;
            z[k] = rd[k] * (r[k] - R.masked(k, lower[k]));
            R.put(i, 0, z[k]);
        }
    }
    for (int c = C - 2; c >= 0; --c)
    {
        tm.sync();
        if (tm.dead()) return;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (col[k] != c) continue;
            const int i = threadIdx.x + k * kTeamThreads;
            z[k] = z[k] - rd[k] * R.masked(k, upper[k]);
            if (c > 0) R.put(i, 0, z[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) rz[k][0] = r[k] * z[k];
}

struct CgScalars
{
    double alpha, beta;
    int go;
};

/// CG of Matrix.cpp:153-222, preconditioned by D^-1 or the multicolour DIC
template <int K, class Team, bool kDic, class Mat>
__global__ void __launch_bounds__(kTeamThreads, 1) k_pers_cg(PersCg<Mat> a, PersArgs t)
{
    __shared__ TeamSmem smem;
    extern __shared__ __align__(16) unsigned char dyn[];
    Team tm(smem, t.g);
    const int n = a.A.n(), lo = min(n, tm.rank * t.chunk), cnt = min(n - lo, t.chunk);
    if (tm.dead())
    {
        tm.finish();
        return;
    }
    if constexpr (Mat::checked)
        if (t.wide && too_wide(tm, a.A, lo, cnt, t.wide))
        {
            tm.finish();
            return;
        }
    Resident<K, 1, Team, resident_regs(K, 1, !kDic)> R(dyn, V3P{{a.g, a.g, a.g}}, lo, cnt);
    R.load(a.A, t.chunk, tm.rank);
    const bool two = t.normType != 0;
    __shared__ CgScalars sc;
    unsigned long long none[1] = {0};
    double x[K], r[K], p[K], d[K], z[K];
    int col[K];
    unsigned lower[K], upper[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const int i = threadIdx.x + k * kTeamThreads;
        const bool in = i < cnt;
        x[k] = in ? a.x[lo + i] : 0.0;
        p[k] = 0.0;
        col[k] = -1;
        lower[k] = upper[k] = 0;
        if constexpr (kDic)
        {
            d[k] = in ? __ldg(a.rDinv + lo + i) : 0.0;
            if (in)
            {
                const int c = lo + i;
                col[k] = __ldg(a.colour + c);
                const long long e0 = a.A.first(c), e1 = a.A.end(c);
                for (int j = 0; j < kResW && e0 + Mat::step * j < e1; ++j)
                {
                    const int cj = a.A.col(e0 + Mat::step * j);
                    if (cj < 0) break;
                    const int oc = __ldg(a.colour + cj);
                    if (oc < col[k]) lower[k] |= 1u << j;
                    else if (oc > col[k]) upper[k] |= 1u << j;
                }
            }
        }
        else d[k] = in ? inv_diag_cg(a.A.diag(lo + i)) : 0.0;
        R.put(i, 0, x[k]);
    }
    tm.sync();
    // the solve's scalars advance in warp 0; alpha, beta and whether to go on
    // reach the block through sc
    double bn = 0.0, init = 0.0, fin = 0.0, rz = 0.0;
    int it = 0, conv = 0;
    {
        double s[K][3];  // r.z, r.r, b.b
        unsigned long long m[2] = {0, 0};  // |r|, |b|
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            const int i = threadIdx.x + k * kTeamThreads;
            double y[1];
            R.row(k, y);
            const double bi = i < cnt ? __ldg(a.b + lo + i) : 0.0;
            r[k] = i < cnt ? bi - y[0] : 0.0;
            z[k] = d[k] * r[k];
            s[k][0] = r[k] * z[k];
            s[k][1] = r[k] * r[k];
            s[k][2] = bi * bi;
            m[0] = max(m[0], mag_bits(r[k]));
            m[1] = max(m[1], mag_bits(bi));
        }
        tm.reduce(s, m, [&](const double (&v)[5]) {
            init = (isnan(v[3]) || isnan(v[4])) ? NAN : (two ? sqrt(v[1]) : v[3]);
            bn = smax(two ? sqrt(v[2]) : (isnan(v[4]) ? 0.0 : v[4]), 1e-300);
            rz = v[0];
            bool go = t.maxIter > 0;
            if (init / bn < t.tol)
            {
                conv = 1;
                fin = init;
                go = false;
            }
            if (threadIdx.x == 0)
            {
                sc.go = go;
                sc.beta = 0.0;
            }
        });
    }
    bool go = sc.go && !tm.dead();
    if constexpr (kDic)
    {
        if (go)
        {
            // the gather vector held x until here
#pragma unroll
            for (int k = 0; k < K; ++k) R.put(threadIdx.x + k * kTeamThreads, 0, z[k]);
            tm.sync();
            double s[K][1] = {};
            pers_dic<K>(tm, R, a.nColours, r, d, col, lower, upper, z, s);
            tm.reduce(s, none, [&](const double (&v)[2]) { rz = v[0]; });
            go = !tm.dead();
        }
    }
    while (go)
    {
        // p = z + beta p (the first iteration's p is 0), for the neighbours too
        const double beta = sc.beta;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            p[k] = z[k] + beta * p[k];
            R.put(threadIdx.x + k * kTeamThreads, 0, p[k]);
        }
        tm.sync();
        if (tm.dead()) break;
        double q[K], s1[K][1];
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            double y[1];
            R.row(k, y);
            q[k] = y[0];
            s1[k][0] = p[k] * y[0];
        }
        tm.reduce(s1, none, [&](const double (&v)[2]) {
            const double alpha = rz / v[0];
            if (threadIdx.x == 0)
            {
                sc.go = !(v[0] <= 0 || fabs(rz) < 1e-300);
                sc.alpha = alpha;
            }
        });
        if (tm.dead() || !sc.go) break;
        const double alpha = sc.alpha;
        double s2[K][2];  // r.z, r.r
        unsigned long long m[1] = {0};
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            x[k] = x[k] + alpha * p[k];
            r[k] = r[k] - alpha * q[k];
            z[k] = d[k] * r[k];
            if constexpr (kDic) R.put(threadIdx.x + k * kTeamThreads, 0, z[k]);
            s2[k][0] = kDic ? 0.0 : r[k] * z[k];
            s2[k][1] = r[k] * r[k];
            m[0] = max(m[0], mag_bits(r[k]));
        }
        tm.reduce(s2, m, [&](const double (&v)[3]) {
            fin = isnan(v[2]) ? NAN : (two ? sqrt(v[1]) : v[2]);
            // lane 0 forms the test's quotient, lane 1 beta
            const bool odd = threadIdx.x & 1;
            const double quot = (odd ? v[0] : fin) / (odd ? rz : bn);
            const double rel = __shfl_sync(0xffffffffu, quot, 0), beta = __shfl_sync(0xffffffffu, quot, 1);
            ++it;
            bool more = false;
            if (rel < t.tol) conv = 1;
            else if (isnan(fin)) it = t.maxIter;
            else more = it < t.maxIter;
            if (!kDic) rz = v[0];
            if (threadIdx.x == 0)
            {
                sc.go = more;
                if (!kDic) sc.beta = beta;
            }
        });
        if (tm.dead() || !sc.go) break;
        if constexpr (kDic)
        {
            double s[K][1] = {};
            pers_dic<K>(tm, R, a.nColours, r, d, col, lower, upper, z, s);
            tm.reduce(s, none, [&](const double (&v)[2]) {
                const double beta = v[0] / rz;
                rz = v[0];
                if (threadIdx.x == 0) sc.beta = beta;
            });
            if (tm.dead()) break;
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const int i = threadIdx.x + k * kTeamThreads;
        if (i < cnt && !tm.dead()) a.x[lo + i] = x[k];
    }
    if (tm.rank == 0 && threadIdx.x == 0)
    {
        SolveState* st = t.st;
        st->it[0] = it;
        st->conv[0] = conv;
        st->init[0] = init;
        st->bnorm[0] = bn;
        st->fin[0] = fin;
        st->done[0] = st->allDone = 1;
        if (t.tally)
        {
            t.tally[0] += it;
            t.tally[1] += conv ? 0.0 : 1.0;
        }
    }
    tm.finish();
}

template <class Mat>
struct PersBi
{
    Mat A;
    V3P b, x;
    V3P g;  // a grid team's copy of the gather vector
};

struct BiScalars
{
    double alpha[3], beta[3], omega[3];
    int done[3], special[3], all;
};

/// NC BiCGStab iterations of Matrix.cpp:224-319 in lockstep over one matrix,
/// each component with its own scalars and stopping test (k_bi_*); lane q of
/// warp 0 advances component q's scalars.  With NC = 1 every team of the
/// launch solves the component of its number: the components share only the
/// matrix, so as teams of their own they take a third of the gathers and of
/// the reduction each, and none waits for another that needs more iterations.
template <int K, class Team, int NC, class Mat>
__global__ void __launch_bounds__(kTeamThreads, 1) k_pers_bicg(PersBi<Mat> a, PersArgs t)
{
    __shared__ TeamSmem smem;
    __shared__ BiScalars sc;
    extern __shared__ __align__(16) unsigned char dyn[];
    Team tm(smem, t.g);
    const int q0 = NC == 1 ? tm.team : 0;  // the team's first component
    const int n = a.A.n(), lo = min(n, tm.rank * t.chunk), cnt = min(n - lo, t.chunk);
    Resident<K, NC, Team, resident_regs(K, NC, false)> R(dyn, NC == 1 ? V3P{{a.g.c[q0], a.g.c[q0], a.g.c[q0]}} : a.g, lo, cnt);
    R.load(a.A, t.chunk, tm.rank);
    const int lane = threadIdx.x & 31, mine = lane < NC ? lane : 0;  // the component this lane advances (warp 0)
    unsigned long long none[1] = {0};
    constexpr bool kXs = resident_xs(K, NC);
    double xr[kXs ? 1 : K][NC];
    double* const xsm = reinterpret_cast<double*>(dyn + resident_smem(K, NC, false)) - (kXs ? NC * K * kTeamThreads : 0);
    auto X = [&](int k, int q) -> double& {
        if constexpr (kXs) return xsm[q * K * kTeamThreads + threadIdx.x + k * kTeamThreads];
        else return xr[k][q];
    };
    double r[K][NC], r0[K][NC], p[K][NC], v[K][NC], id[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const int i = threadIdx.x + k * kTeamThreads;
        id[k] = i < cnt ? inv_diag_bicg(a.A.diag(lo + i)) : 0.0;
#pragma unroll
        for (int q = 0; q < NC; ++q)
        {
            X(k, q) = i < cnt ? a.x.c[q0 + q][lo + i] : 0.0;
            p[k][q] = v[k][q] = 0.0;
            R.put(i, q, X(k, q));
        }
    }
    tm.sync();
    // this lane's component
    double bn = 0.0, init = 0.0, fin = 0.0, rho = 1.0, alpha = 1.0, omega = 1.0, rz = 0.0;
    int it = 0, conv = 0, done = 0;
    // value q of this lane's component from the values of a reduction
    auto pick = [&](const double* w) {
        double o = w[0];
#pragma unroll
        for (int q = 1; q < NC; ++q)
            if (mine == q) o = w[q];
        return o;
    };
    auto publish = [&]() {
        const unsigned ds = __ballot_sync(0xffffffffu, done != 0) & ((1u << NC) - 1u);
        if (lane < NC) sc.done[lane] = done;
        if (lane == 0) sc.all = ds == (1u << NC) - 1u;
    };
    {
        double s[K][NC];
        unsigned long long m[2 * NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) m[q] = m[NC + q] = 0;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            const int i = threadIdx.x + k * kTeamThreads;
            double y[NC];
            R.row(k, y);
#pragma unroll
            for (int q = 0; q < NC; ++q)
            {
                const double bi = i < cnt ? a.b.c[q0 + q][lo + i] : 0.0;
                r[k][q] = r0[k][q] = i < cnt ? bi - y[q] : 0.0;
                m[q] = max(m[q], mag_bits(r[k][q]));
                m[NC + q] = max(m[NC + q], mag_bits(bi));
                s[k][q] = r[k][q] * r[k][q];
            }
        }
        tm.reduce(s, m, [&](const double (&w)[3 * NC]) {
            rz = pick(w);
            const double rInf = pick(w + NC), bInf = pick(w + 2 * NC);
            init = (isnan(rInf) || isnan(bInf)) ? NAN : rInf;
            bn = smax(isnan(bInf) ? 0.0 : bInf, 1e-300);
            conv = init / bn < t.tol;
            fin = conv ? init : 0.0;
            done = conv || t.maxIter <= 0 || fabs(rz) < 1e-300;
            if (lane < NC)
            {
                sc.beta[lane] = rz;  // (rz / rho) (alpha / omega), all 1
                sc.omega[lane] = 1.0;
            }
            publish();
        });
    }
    while (!sc.all && !tm.dead())
    {
        // p = r + beta (p - omega v); z = p D^-1 for the neighbours
#pragma unroll
        for (int q = 0; q < NC; ++q)
        {
            const double be = sc.beta[q], om = sc.omega[q];
            const bool dn = sc.done[q];
#pragma unroll
            for (int k = 0; k < K; ++k)
            {
                if (!dn) p[k][q] = r[k][q] + be * (p[k][q] - om * v[k][q]);
                R.put(threadIdx.x + k * kTeamThreads, q, p[k][q] * id[k]);
            }
        }
        tm.sync();
        if (tm.dead()) break;
        // v = A z; r0.v; alpha
        double sv[K][NC];
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            R.row(k, v[k]);
#pragma unroll
            for (int q = 0; q < NC; ++q) sv[k][q] = r0[k][q] * v[k][q];
        }
        tm.reduce(sv, none, [&](const double (&w)[NC + 1]) {
            const double den = pick(w);
            if (!done)
            {
                rho = rz;
                if (fabs(den) < 1e-300) done = 1;
                else alpha = rho / den;
            }
            if (lane < NC) sc.alpha[lane] = alpha;
            publish();
        });
        if (tm.dead() || sc.all) break;
        // s = r - alpha v into r; sh = s D^-1 for the neighbours
#pragma unroll
        for (int q = 0; q < NC; ++q)
        {
            const double al = sc.alpha[q];
            const bool dn = sc.done[q];
#pragma unroll
            for (int k = 0; k < K; ++k)
            {
                if (!dn) r[k][q] = r[k][q] - al * v[k][q];
                R.put(threadIdx.x + k * kTeamThreads, q, r[k][q] * id[k]);
            }
        }
        tm.sync();
        if (tm.dead()) break;
        // t = A sh; t.t and t.s; omega, or the breakdown exit
        double tv[K][NC], st[K][2 * NC];
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            R.row(k, tv[k]);
#pragma unroll
            for (int q = 0; q < NC; ++q)
            {
                st[k][q] = tv[k][q] * tv[k][q];
                st[k][NC + q] = tv[k][q] * r[k][q];
            }
        }
        tm.reduce(st, none, [&](const double (&w)[2 * NC + 1]) {
            const double den = pick(w), num = pick(w + NC);
            int special = 0;
            if (!done)
            {
                if (den < 1e-300)
                {
                    special = done = 1;
                    ++it;
                }
                else omega = num / den;
            }
            if (lane < NC)
            {
                sc.omega[lane] = omega;
                sc.special[lane] = special;
                sc.done[lane] = done;
            }
        });
        if (tm.dead()) break;
        // x = (x + alpha z) + omega sh; r = s - omega t; |r|inf; next r0.r
        double sr[K][NC];
        unsigned long long m[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q)
        {
            m[q] = 0;
            const double al = sc.alpha[q], om = sc.omega[q];
            const bool dn = sc.done[q], sp = sc.special[q];
#pragma unroll
            for (int k = 0; k < K; ++k)
            {
                sr[k][q] = 0.0;
                if (sp) X(k, q) = X(k, q) + al * (p[k][q] * id[k]);
                else if (!dn)
                {
                    X(k, q) = (X(k, q) + al * (p[k][q] * id[k])) + om * (r[k][q] * id[k]);
                    r[k][q] = r[k][q] - om * tv[k][q];
                    sr[k][q] = r0[k][q] * r[k][q];
                }
                m[q] = max(m[q], mag_bits(r[k][q]));
            }
        }
        tm.reduce(sr, m, [&](const double (&w)[2 * NC]) {
            const double rNew = pick(w), rInf = pick(w + NC);
            // three quotients per component, one per lane group: the test's,
            // rz / rho and alpha / omega
            const int g = lane < 8 ? 0 : (lane < 16 ? 1 : 2);
            const int src = lane & 7;
            const double n0 = __shfl_sync(0xffffffffu, rInf, src), n1 = __shfl_sync(0xffffffffu, rNew, src),
                         n2 = __shfl_sync(0xffffffffu, alpha, src);
            const double d0 = __shfl_sync(0xffffffffu, bn, src), d1 = __shfl_sync(0xffffffffu, rho, src),
                         d2 = __shfl_sync(0xffffffffu, omega, src);
            const double quot = (g == 0 ? n0 : (g == 1 ? n1 : n2)) / (g == 0 ? d0 : (g == 1 ? d1 : d2));
            const double rel = __shfl_sync(0xffffffffu, quot, src), f1 = __shfl_sync(0xffffffffu, quot, 8 + src),
                         f2 = __shfl_sync(0xffffffffu, quot, 16 + src);
            const int special = lane < NC ? sc.special[lane] : 0;
            if (special)
            {
                fin = rInf;
                conv = rel < t.tol;
            }
            else if (!done)
            {
                ++it;
                fin = rInf;
                if (rel < t.tol) conv = done = 1;
                else if (isnan(fin))
                {
                    it = t.maxIter;
                    done = 1;
                }
                else
                {
                    rz = rNew;
                    if (it >= t.maxIter || fabs(rNew) < 1e-300) done = 1;
                }
            }
            if (lane < NC) sc.beta[lane] = f1 * f2;
            publish();
        });
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const int i = threadIdx.x + k * kTeamThreads;
        if (i < cnt && !tm.dead())
#pragma unroll
            for (int q = 0; q < NC; ++q) a.x.c[q0 + q][lo + i] = X(k, q);
    }
    if (tm.rank == 0 && threadIdx.x < 32)
    {
        SolveState* o = t.st;
        if (lane < NC)
        {
            o->it[q0 + lane] = it;
            o->conv[q0 + lane] = conv;
            o->init[q0 + lane] = init;
            o->bnorm[q0 + lane] = bn;
            o->fin[q0 + lane] = fin;
            o->done[q0 + lane] = 1;
        }
        int its = lane < NC ? it : 0, open = lane < NC && !conv;
#pragma unroll
        for (int s = 2; s > 0; s >>= 1)
        {
            its += __shfl_down_sync(0xffffffffu, its, s);
            open += __shfl_down_sync(0xffffffffu, open, s);
        }
        if (lane == 0)
        {
            o->allDone = 1;
            if (t.tally)
            {
                atomicAdd(t.tally, static_cast<double>(its));  // whole numbers: any order
                atomicAdd(t.tally + 1, static_cast<double>(open));
            }
        }
    }
    tm.finish();
}

// ---- host side ----------------------------------------------------------------

// rows per thread that registers and shared memory hold: one component, and
// the three-component BiCGStab
constexpr int kRes1K = kTeamRowsMax, kRes3K = 2;

/// f(std::integral_constant<int, K>) for 1 <= K <= Kmax
template <int Kmax, class F>
void dispatchK(int K, F&& f)
{
    if constexpr (Kmax > 1)
        if (K < Kmax) return dispatchK<Kmax - 1>(K, f);
    f(std::integral_constant<int, Kmax>{});
}

inline TeamMem teamMem(const TeamPlan& tp, int n, unsigned* count, double* part, int* failed, long long start = 0)
{
    return TeamMem{tp.blocks, count, part, (n + kGroupRows - 1) / kGroupRows, tp.chunk / kGroupRows, failed,
                   teamWaitLimit(), start};
}
/// doubles of `part` for a system of n rows in one team, and in any plan
constexpr size_t teamPartMax(int n) { return 2 * kTeamVals * (static_cast<size_t>(n) / kGroupRows + 1); }
inline size_t teamPartSize(int n) { return kTeamsMax * 2 * kTeamVals * (static_cast<size_t>(n) / kGroupRows + 1); }

/// A whole-solve kernel as `teams` teams of the plan on stream s.
template <class Kern, class A>
void launchTeam(const TeamPlan& tp, int teams, Kern kernel, const A& args, const PersArgs& t, size_t smem, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tp.blocks * teams));
    cfg.blockDim = dim3(kTeamThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    CFG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (tp.cluster)
    {
        if (tp.blocks > 8) CFG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = static_cast<unsigned>(tp.blocks);
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    }
    else if (t.g.start == 0)
    {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = tp.cluster || t.g.start == 0 ? 1 : 0;
    CFG_CUDA(cudaLaunchKernelEx(&cfg, kernel, args, t));
}

}  // namespace cfg
