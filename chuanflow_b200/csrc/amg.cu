// Aggregation-AMG preconditioner for the pressure equation, in FP32 inside
// the FP64 flexible CG (no reference counterpart: the reference solves its
// pressure with Jacobi-PCG, Matrix.cpp:153-222).
//
// Structure (host, once per mesh): aggregation of the matrix graph in
// device numbering.  Phase 1 visits rows in order and makes a row whose
// neighbours are all free the root of an aggregate of itself and those
// neighbours; phase 2 puts every row left over into the aggregate of its
// first aggregated neighbour.  Plain aggregation counts every entry as a
// neighbour; with strength of connection (the pressure hierarchy when its
// threshold is set) only the strong entries count.  The momentum matrix
// has a hierarchy of its own, aggregated plainly.  The coarse operator is
// the Galerkin product P^T A P with the piecewise-constant P, so every
// coarse entry is a plain sum of fine entries: the host lists, per coarse
// entry, the fine entries it sums (in a fixed order), and the device forms
// the values with one gather kernel per level.  Levels stop at <= 128 rows, whose operator is inverted
// densely on the host (diagonally regularised when singular, as a pure
// Neumann system is).
//
// V-cycle (device, FP32 vectors and values): on the finest level one kernel
// does a damped-Jacobi sweep from zero and the residual; the residual is
// summed over each aggregate; the coarse levels sweep, correct and sweep
// again, one to four weighted sweeps each time (smootherOf); a correction is
// scaled by s > 1, which makes up for the piecewise constant interpolation;
// and one kernel does the finest level's last sweep.  The finest level reads
// the FCG residual in FP64 and writes z in FP64.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <mutex>
#include <numeric>
#include <type_traits>
#include <utility>
#include <vector>

#include "ctx.h"
#include "kernels.cuh"

namespace cfg
{

/// m Jacobi sweeps and their weights: w[0], w[1], ... before a coarse
/// correction, in reverse after it.
constexpr int kSweepsMax = 4;
struct Sweeps
{
    int m = 1;
    float w[kSweepsMax] = {};
};

/// The sweeps of the first coarse level and of the levels below it (the
/// finest has one of weight kOmega on either side).
struct Smoother
{
    Sweeps first, rest;
    const Sweeps& at(int level) const { return level <= 1 ? first : rest; }
};

struct AmgLevel
{
    int n = 0;
    // levels >= 1 below the coarsest: CSR operator, diagonal position per row
    int *rs = nullptr, *cols = nullptr, *dpos = nullptr;
    float* val = nullptr;
    float* dinv = nullptr;
    // to the next level: the aggregate of each row, each aggregate's rows,
    // and per next-level entry the entries of this level it sums
    int* agg = nullptr;
    int *ms = nullptr, *mem = nullptr;
    int *gs = nullptr, *gl = nullptr;
    int nnzNext = 0;
    // lanes per row of this level's passes (levels >= 1) and per aggregate
    // of its restriction into the next level
    int gRow = 4, gAgg = 4;
    // a large coarse level's operator also as SELL-32 (one thread per row):
    // slice starts, columns (-1 on the pads) and values, and per CSR entry
    // its SELL position; sstart null: the level's passes use lane groups
    int *sstart = nullptr, *scol = nullptr, *sellPos = nullptr;
    float* sval = nullptr;
    // work vectors: rhs, first sweep, residual, output
    float *b = nullptr, *x = nullptr, *r = nullptr, *xo = nullptr;
    // the same for the three-component V-cycle (a float4 per row), allocated
    // on its first use
    float *b3 = nullptr, *x3 = nullptr, *r3 = nullptr, *xo3 = nullptr;
};

/// Device scalars of the device-resident flexible CG (amgFcg)
struct FcgState
{
    double tol, bn, pq, alpha, beta, rn, init;
    int it, maxIter, done, conv;
    int normType;  // 1: |r|2 / |b|2 <= tol; 0: |r|inf / max(|b|inf, 1e-300) < tol (the reference's test)
    unsigned int ticket[4];
};

struct AmgState
{
    ~AmgState()
    {
        for (auto& g : graphs) cudaGraphExecDestroy(g.second);
        if (stHost) cudaFreeHost(stHost);
    }
    // (values, solution vector, chunk) -> graph
    std::vector<std::pair<std::pair<std::pair<const void*, const void*>, int>, cudaGraphExec_t>> graphs;
    FcgState* st = nullptr;
    FcgState* stHost = nullptr;
    std::vector<AmgLevel> lv;
    int nc = 0;                  // rows of the coarsest level (dense inverse)
    float* dense = nullptr;      // nc x nc inverse
    std::vector<int> hrs, hcols;  // coarsest CSR on the host
    bool valuesReady = false;
    double setupMs = 0, valuesMs = 0;
    double theta = 0;                 // strength threshold of the aggregation (0: plain)
    const float* vals32 = nullptr;    // the finest operator's FP32 SELL values
    // k_amg_tail: the dynamic shared memory of the last aggregated level and
    // its entries (0: it does not fit, its kernels and k_amg_dense run)
    size_t tailSmem = 0;
    int tailNnz = 0;
    bool tailCluster = false;  // k_amg_tail, else k_amg_tail_block
    bool decoupled = false;  // the strong entries leave next to nothing between the aggregates
    int skewClass = 0;    // how far from symmetric the finest operator is (skewOf)
    double* skew = nullptr;
};

void AmgDeleter::operator()(AmgState* a) const { delete a; }

namespace
{

constexpr float kOmega = 0.8f;    // damped Jacobi
constexpr float kScale = kAmgScalePressure;  // coarse-correction scaling of the single V-cycle
constexpr int kDenseMax = 128;
// coarse levels of at least this many rows keep a SELL-32 copy of their
// operator: one thread per row fills the GPU in one wave there
constexpr int kSellMinRows = 32768;

// first coarse levels of this many rows or more take four sweeps, not three
// (smootherOf)
constexpr int kFourMinRows = 100000;

/// m sweeps whose product is the Chebyshev polynomial of [lo, hi] in D^-1 A
Sweeps chebyshev(int m, double lo, double hi)
{
    Sweeps s;
    s.m = m;
    for (int k = 0; k < m; ++k)
        s.w[k] = static_cast<float>(1.0 / (0.5 * (hi + lo) + 0.5 * (hi - lo) * std::cos(M_PI * (2 * k + 1) / (2.0 * m))));
    return s;
}
Sweeps jacobi(int m)
{
    Sweeps s;
    s.m = m;
    for (int k = 0; k < m; ++k) s.w[k] = kOmega;
    return s;
}
/// one sweep before and after each correction on every level
Smoother singleSweeps() { return Smoother{jacobi(1), jacobi(1)}; }

constexpr int kSingleSweeps = 2;  // the class whose V-cycle has one sweep on every level
/// The class of a nonsymmetric operator by theta = max over rows of
/// sum_j |a_ij - a_ji| / (2 a_ii), a bound of the imaginary parts of D^-1 A:
/// Chebyshev sweeps amplify eigenvalues far off the real axis.
int skewOf(double theta) { return theta <= 0.5 ? 0 : (theta <= 0.7 ? 1 : kSingleSweeps); }

/// One full wave of a grid-stride row kernel of TPB threads: the SMs times
/// the blocks of this kernel one SM holds at once (its registers decide),
/// at most one block per TPB rows.  The finest-level V-cycle passes and the
/// FCG's SpMV are bound by the latency of their gathers (each waits on the
/// column loaded before it), so every warp slot an SM has is filled; the
/// count is looked up once per kernel.
int waveGrid(const void* kernel, int sms, int rows)
{
    static std::mutex mu;
    static std::vector<std::pair<const void*, int>> perSM;
    int per = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        for (const auto& k : perSM)
            if (k.first == kernel) per = k.second;
        if (per == 0)
        {
            CFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, TPB, 0));
            per = std::max(1, per);
            perSM.push_back({kernel, per});
        }
    }
    return std::max(1, std::min((rows + TPB - 1) / TPB, sms * per));
}

/// f(std::integral_constant<int, G>{}) for the lane group g (4, 8, 16 or 32)
template <class F>
void withGroup(int g, F&& f)
{
    switch (g)
    {
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        case 32: f(std::integral_constant<int, 32>{}); break;
        default: f(std::integral_constant<int, 4>{}); break;
    }
}

/// one SELL row of the finest operator: sum over its entries of val * f(col).
/// W bounds the row length at compile time: all columns and values of the
/// row are loaded before the first gather (W = 0 walks any length).
template <int W, class F>
__device__ __forceinline__ float sell_row(const DMat& A, const float* __restrict__ val, int c, F f)
{
    const int sl = c >> 5, lane = c & 31;
    const int e0 = __ldg(A.start + sl) + lane, e1 = __ldg(A.start + sl + 1);
    float s = 0.0f;
    if constexpr (W > 0)
    {
        int col[W];
        float v[W];
#pragma unroll
        for (int k = 0; k < W; ++k)
        {
            const int e = e0 + 32 * k;
            col[k] = e < e1 ? __ldg(A.col + e) : -1;
            v[k] = e < e1 ? __ldg(val + e) : 0.0f;
        }
        float g[W];
#pragma unroll
        for (int k = 0; k < W; ++k) g[k] = col[k] >= 0 ? f(col[k]) : 0.0f;
#pragma unroll
        for (int k = 0; k < W; ++k) s += v[k] * g[k];
    }
    else
    {
        for (int e = e0; e < e1; e += 32)
        {
            const int col = __ldg(A.col + e);
            if (col < 0) break;
            s += __ldg(val + e) * f(col);
        }
    }
    return s;
}

/// finest level, first sweep and residual: x = w D^-1 b, r = b - A x
template <int W>
__global__ void __launch_bounds__(TPB) k_amg_pre0(const int* stop, DMat A, const float* __restrict__ val,
                                                  const float* __restrict__ dinv, const double* b,
                                                  float* __restrict__ x, float* __restrict__ r)
{
    pdl_entry();
    if (stop && *stop) return;
    FOR_ROWS(c, A.n)
    {
        const float bc = static_cast<float>(b[c]);
        x[c] = kOmega * dinv[c] * bc;
        const float s =
            sell_row<W>(A, val, c, [&](int j) { return kOmega * __ldg(dinv + j) * static_cast<float>(b[j]); });
        r[c] = bc - s;
    }
}

/// finest level: z = y + w D^-1 (b - A y), in FP64 out; inside the device
/// FCG (st given) also z.q and, in the block that finishes last,
/// beta = -z.q / p.q
template <int W>
__global__ void __launch_bounds__(TPB) k_amg_post0(const int* stop, DMat A, const float* __restrict__ val,
                                                   const float* __restrict__ dinv, const double* b, const float* y,
                                                   double* __restrict__ z, const double* q, double* partials,
                                                   FcgState* st)
{
    pdl_entry();
    if (stop && *stop) return;
    const bool dot = q != nullptr;  // inside the FCG iteration
    double zq[1] = {0.0};
    FOR_ROWS(c, A.n)
    {
        const float s = sell_row<W>(A, val, c, [&](int j) { return y[j]; });
        const double zc = static_cast<double>(y[c] + kOmega * dinv[c] * (static_cast<float>(b[c]) - s));
        z[c] = zc;
        if (dot) zq[0] += zc * q[c];
    }
    if (!dot) return;
    block_sum<1>(zq);
    if (threadIdx.x == 0) partials[blockIdx.x] = zq[0];
    if (!last_block(&st->ticket[2])) return;
    double f[1];
    final_sum<1>(partials, gridDim.x, f);
    if (threadIdx.x == 0)
    {
        st->ticket[2] = 0;
        st->beta = -f[0] / st->pq;
    }
}

/// next-level entries as sums of this level's: FP64 sums of FP64 (finest,
/// SELL) or FP32 values, stored in FP32
__global__ void __launch_bounds__(TPB) k_amg_galerkin(int nnz, const int* __restrict__ gs, const int* __restrict__ gl,
                                                      const double* __restrict__ fineD, const float* __restrict__ fineF,
                                                      float* __restrict__ out)
{
    FOR_ROWS(e, nnz)
    {
        double s = 0.0;
        for (int k = gs[e]; k < gs[e + 1]; ++k) s += fineD ? fineD[gl[k]] : static_cast<double>(fineF[gl[k]]);
        out[e] = static_cast<float>(s);
    }
}

/// max over rows of sum_j |a_ij - a_ji| / (2 a_ii), into the bits of *out; a
/// row with a NaN counts as 1e300
__global__ void __launch_bounds__(TPB) k_amg_skew(DMat A, const double* __restrict__ val, unsigned long long* out)
{
    double mx[1] = {0.0};
    FOR_ROWS(i, A.n)
    {
        const int e1 = __ldg(A.start + (i >> 5) + 1);
        double s = 0.0, d = 0.0;
        for (int e = __ldg(A.start + (i >> 5)) + (i & 31); e < e1; e += 32)
        {
            const int j = __ldg(A.col + e);
            if (j < 0) break;
            const double v = __ldg(val + e);
            if (j == i)
            {
                d = v;
                continue;
            }
            double w = 0.0;
            const int f1 = __ldg(A.start + (j >> 5) + 1);
            for (int f = __ldg(A.start + (j >> 5)) + (j & 31); f < f1; f += 32)
            {
                const int c = __ldg(A.col + f);
                if (c < 0) break;
                if (c == i)
                {
                    w = __ldg(val + f);
                    break;
                }
            }
            s += fabs(v - w);
        }
        const double t = d > 0.0 ? s / (2.0 * d) : 1.0;
        mx[0] = smax(mx[0], isnan(t) ? 1e300 : t);  // a NaN counts as the worst
    }
    block_max<1>(mx);
    if (threadIdx.x == 0) atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(mx[0])));
}

__global__ void __launch_bounds__(TPB) k_amg_dinv(int n, const int* __restrict__ dpos, const float* __restrict__ val,
                                                  float* __restrict__ dinv)
{
    FOR_ROWS(i, n)
    {
        const float d = val[dpos[i]];
        dinv[i] = d != 0.0f ? 1.0f / d : 1.0f;
    }
}

__global__ void __launch_bounds__(TPB) k_amg_dinv0(int n, const double* __restrict__ diag, float* __restrict__ dinv)
{
    FOR_ROWS(i, n) dinv[i] = diag[i] != 0.0 ? static_cast<float>(1.0 / diag[i]) : 1.0f;
}

// ---- the V-cycle on three right-hand sides at once (the momentum
// components share their matrix): the same arithmetic per component as the
// single V-cycle above, with the matrix read once for the three.  `done`
// (the BiCGStab's per-component flags) zeroes a converged component's input
// lanes and leaves its output z_q as it was; the V-cycle returns at once
// when all three are done.

/// one SELL row of the finest operator against three vectors
template <int W, class F>
__device__ __forceinline__ void sell_row3(const DMat& A, const float* __restrict__ val, int c, float (&s)[3], F f)
{
    const int sl = c >> 5, lane = c & 31;
    const int e0 = __ldg(A.start + sl) + lane, e1 = __ldg(A.start + sl + 1);
    s[0] = s[1] = s[2] = 0.0f;
    if constexpr (W > 0)
    {
        constexpr int CH = W > 8 ? 8 : W;
#pragma unroll
        for (int k0 = 0; k0 < W; k0 += CH)
        {
            int col[CH];
            float v[CH];
#pragma unroll
            for (int k = 0; k < CH; ++k)
            {
                const int e = e0 + 32 * (k0 + k);
                col[k] = (k0 + k < W && e < e1) ? __ldg(A.col + e) : -1;
                v[k] = (k0 + k < W && e < e1) ? __ldg(val + e) : 0.0f;
            }
            float g[CH][3];
#pragma unroll
            for (int k = 0; k < CH; ++k)
            {
                if (col[k] >= 0) f(col[k], g[k]);
                else g[k][0] = g[k][1] = g[k][2] = 0.0f;
            }
#pragma unroll
            for (int k = 0; k < CH; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) s[q] += v[k] * g[k][q];
        }
    }
    else
    {
        for (int e = e0; e < e1; e += 32)
        {
            const int col = __ldg(A.col + e);
            if (col < 0) break;
            float g[3];
            f(col, g);
            const float v = __ldg(val + e);
#pragma unroll
            for (int q = 0; q < 3; ++q) s[q] += v * g[q];
        }
    }
}

struct Active3
{
    bool a[3];
    __device__ bool none() const { return !(a[0] || a[1] || a[2]); }
};
__device__ __forceinline__ Active3 active3(const int* done)
{
    return Active3{{done[0] == 0, done[1] == 0, done[2] == 0}};
}

// Level vectors of the three-component V-cycle hold one float4 per row: the
// three components in x, y, z (w is zero).  A row gathered by a neighbour's
// sweep or by its aggregate's restriction is one 16-byte load, not three
// scattered ones.  A converged component's lanes carry zeros (its input lanes
// are read as zero), so every lane is computed and stored.

__device__ __forceinline__ float4 pack3(const float (&v)[3]) { return make_float4(v[0], v[1], v[2], 0.0f); }
__device__ __forceinline__ void unpack3(float4 p, float (&v)[3])
{
    v[0] = p.x;
    v[1] = p.y;
    v[2] = p.z;
}

/// finest level, first sweep and residual for three FP64 right-hand sides:
/// x = w D^-1 b and r = b - A x
template <int W>
__global__ void __launch_bounds__(TPB, (W > 0 && W <= 8) ? 6 : 1) k_amgv_pre0(const int* done, DMat A, const float* __restrict__ val,
                                                   const float* __restrict__ dinv, CV3P b, float4* __restrict__ x,
                                                   float4* __restrict__ r)
{
    pdl_entry();
    const Active3 act = active3(done);
    if (act.none()) return;
    const int n = A.n;
    FOR_ROWS(c, n)
    {
        float s[3];
        sell_row3<W>(A, val, c, s, [&](int j, float (&g)[3]) {
            const float wd = kOmega * __ldg(dinv + j);
#pragma unroll
            for (int q = 0; q < 3; ++q) g[q] = act.a[q] ? wd * static_cast<float>(b.c[q][j]) : 0.0f;
        });
        const float dc = dinv[c];
        float xv[3], rv[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
            const float bc = act.a[q] ? static_cast<float>(b.c[q][c]) : 0.0f;
            xv[q] = kOmega * dc * bc;
            rv[q] = bc - s[q];
        }
        x[c] = pack3(xv);
        r[c] = pack3(rv);
    }
}

/// finest level: z = y + w D^-1 (b - A y), into FP64 (active components only)
template <int W>
__global__ void __launch_bounds__(TPB) k_amgv_post0(const int* done, DMat A, const float* __restrict__ val,
                                                    const float* __restrict__ dinv, CV3P b, const float4* y,
                                                    V3P z)
{
    pdl_entry();
    const Active3 act = active3(done);
    if (act.none()) return;
    const int n = A.n;
    FOR_ROWS(c, n)
    {
        float s[3];
        sell_row3<W>(A, val, c, s, [&](int j, float (&g)[3]) { unpack3(y[j], g); });
        const float dc = dinv[c];
        float yc[3];
        unpack3(y[c], yc);
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (act.a[q])
                z.c[q][c] = static_cast<double>(yc[q] + kOmega * dc * (static_cast<float>(b.c[q][c]) - s[q]));
    }
}

// ---- the coarse levels, for one vector (V float) or three at once (V
// float4, a component per lane of it): the same arithmetic and orders per
// component, so the three-vector V-cycle gives each component the single
// one's bits

__device__ __forceinline__ void vzero(float& v) { v = 0.0f; }
__device__ __forceinline__ void vzero(float4& v) { v = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
__device__ __forceinline__ void vmad(float& s, float a, float v) { s += a * v; }
__device__ __forceinline__ void vmad(float4& s, float a, float4 v)
{
    s.x += a * v.x;
    s.y += a * v.y;
    s.z += a * v.z;
}
__device__ __forceinline__ float vscaled(float a, float v) { return a * v; }
__device__ __forceinline__ float4 vscaled(float a, float4 v) { return make_float4(a * v.x, a * v.y, a * v.z, 0.0f); }
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float4 vadd(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, 0.0f); }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ float4 vsub(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, 0.0f); }
template <int G>
__device__ __forceinline__ void vgroup(float& s)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
}
template <int G>
__device__ __forceinline__ void vgroup(float4& s)
{
    vgroup<G>(s.x);
    vgroup<G>(s.y);
    vgroup<G>(s.z);
}
/// whether a kernel's vectors may still change: the single V-cycle's stop
/// flag, or all three components' done flags
__device__ __forceinline__ bool halted(const int* f, float) { return f && *f; }
__device__ __forceinline__ bool halted(const int* f, float4) { return f[0] && f[1] && f[2]; }

/// A coarse level on the device: its operator, its aggregates' members and
/// its vectors (rhs, first sweep, residual, output).
template <class V>
struct Coarse
{
    int n;
    const int *rs, *cols;
    const float *val, *dinv;
    const int *agg, *ms, *mem;  // to the next level
    const int *sstart, *scol;   // SELL-32 copy (null: none)
    const float* sval;
    V *b, *x, *r, *o;
    int gRow, gAgg;
};

/// Row i summed by a group of G lanes, lane l taking entries l, l + G, ...;
/// the group's lanes hold the sum after the shuffle tree.
template <class V, int G>
__device__ __forceinline__ V group_row(const Coarse<V>& L, int i, int l, const V* x)
{
    V s;
    vzero(s);
    if (i >= 0)
        for (int e = __ldg(L.rs + i) + l; e < __ldg(L.rs + i + 1); e += G)
            vmad(s, __ldg(L.val + e), x[__ldg(L.cols + e)]);
    vgroup<G>(s);
    return s;
}

/// Calls body(i, l) for every row in groups of G lanes; whole warps go round
/// together (the shuffles need every lane), i is -1 past the last row.
template <int G, class F>
__device__ __forceinline__ void group_loop(int n, int thread, int threads, F&& body)
{
    const int l = threadIdx.x % G;
    for (int i0 = thread / G;; i0 += threads / G)
    {
        if (i0 - (threadIdx.x % 32) / G >= n) break;
        body(i0 < n ? i0 : -1, l);
    }
}

/// the residual r of the level above summed over each of this level's n
/// aggregates: its right-hand side b and, dinv given, first sweep x = w D^-1 b
template <class V, int G>
__device__ __forceinline__ void do_restrict(int n, const int* __restrict__ ms, const int* __restrict__ mem, const V* r,
                                            const float* dinv, float w, V* b, V* x, int thread, int threads)
{
    group_loop<G>(n, thread, threads, [&](int I, int l) {
        V s;
        vzero(s);
        if (I >= 0)
            for (int k = __ldg(ms + I) + l; k < __ldg(ms + I + 1); k += G)
                s = vadd(s, r[__ldg(mem + k)]);
        vgroup<G>(s);
        if (I < 0 || l != 0) return;
        b[I] = s;
        if (dinv) x[I] = vscaled(w * dinv[I], s);
    });
}

/// r = b - A x
template <class V, int G>
__device__ __forceinline__ void do_residual(const Coarse<V>& L, const V* x, V* r, int thread, int threads)
{
    group_loop<G>(L.n, thread, threads, [&](int i, int l) {
        const V s = group_row<V, G>(L, i, l, x);
        if (i >= 0 && l == 0) r[i] = vsub(L.b[i], s);
    });
}

/// out = y + w D^-1 (b - A y)
template <class V, int G>
__device__ __forceinline__ void do_smooth(const Coarse<V>& L, float w, const V* y, V* out, int thread, int threads)
{
    group_loop<G>(L.n, thread, threads, [&](int i, int l) {
        const V s = group_row<V, G>(L, i, l, y);
        if (i >= 0 && l == 0) out[i] = vadd(y[i], vscaled(w * L.dinv[i], vsub(L.b[i], s)));
    });
}

template <class V, int G>
__global__ void __launch_bounds__(TPB) k_amg_restrict(const int* stop, int n, const int* __restrict__ ms,
                                                      const int* __restrict__ mem, const V* r,
                                                      const float* __restrict__ dinv, float w, V* __restrict__ b,
                                                      V* __restrict__ x)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    do_restrict<V, G>(n, ms, mem, r, dinv, w, b, x, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}

template <class V, int G>
__global__ void __launch_bounds__(TPB) k_amg_residual(const int* stop, Coarse<V> L, const V* x, V* __restrict__ r)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    do_residual<V, G>(L, x, r, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}

template <class V, int G>
__global__ void __launch_bounds__(TPB) k_amg_smooth(const int* stop, Coarse<V> L, float w, const V* y, V* __restrict__ out)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    do_smooth<V, G>(L, w, y, out, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}

/// the coarse correction brought to a level: y = x + s P xc
template <class V>
__global__ void __launch_bounds__(TPB) k_amg_prolong(const int* stop, int n, const V* x, const V* xc, const int* __restrict__ agg,
                                                     V* __restrict__ y, float scale)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    FOR_ROWS(i, n) y[i] = vadd(x[i], vscaled(scale, xc[agg[i]]));
}

// Large coarse levels in SELL-32, one thread per row: each row summed in its
// CSR column order; columns and values of eight slots are loaded before
// their gathers.

/// a coarse level's CSR values into its SELL-32 copy (the pads stay 0)
__global__ void __launch_bounds__(TPB) k_amg_to_sell(int nnz, const int* __restrict__ pos, const float* __restrict__ val,
                                                     float* __restrict__ sval)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) sval[pos[e]] = val[e];
}

template <class V>
__device__ __forceinline__ V sell32_row(const Coarse<V>& L, int i, const V* x)
{
    const int e0 = __ldg(L.sstart + (i >> 5)) + (i & 31), e1 = __ldg(L.sstart + (i >> 5) + 1);
    V s;
    vzero(s);
    for (int eb = e0; eb < e1; eb += 32 * 8)
    {
        int col[8];
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            const int e = eb + 32 * k;
            col[k] = e < e1 ? __ldg(L.scol + e) : -1;
            v[k] = e < e1 ? __ldg(L.sval + e) : 0.0f;
        }
        V g[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            if (col[k] >= 0) g[k] = x[col[k]];
            else vzero(g[k]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) vmad(s, v[k], g[k]);
    }
    return s;
}

/// r = b - A x
template <class V>
__global__ void __launch_bounds__(TPB) k_amg_residual_sell(const int* stop, Coarse<V> L, const V* x, V* __restrict__ r)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    FOR_ROWS(i, L.n) r[i] = vsub(L.b[i], sell32_row(L, i, x));
}

/// out = y + w D^-1 (b - A y)
template <class V>
__global__ void __launch_bounds__(TPB) k_amg_smooth_sell(const int* stop, Coarse<V> L, float w, const V* y, V* __restrict__ out)
{
    pdl_entry();
    if (halted(stop, V{})) return;
    FOR_ROWS(i, L.n)
    {
        const V s = sell32_row(L, i, y);
        out[i] = vadd(y[i], vscaled(w * L.dinv[i], vsub(L.b[i], s)));
    }
}

// ---- the last levels ----------------------------------------------------------

constexpr int kTailMax = 1024;  // rows of the fused last aggregation level
constexpr int kTailThreads = 1024;
// A cluster per vector above two entries per thread, one block below, where
// a product is a few hundred cycles and the barriers between them would be
// more.  Whole solves, block -> cluster: 55k tets (529 rows, 6,935 entries)
// 2.87 -> 2.64 ms, 1.2M hexahedra (279, 4,725) 16.4 -> 15.8 ms, 2M-cell
// channel (514, 9,450) 158.7 -> 155.4 ms, 262k-cell channel (458, 4,720 and
// 269, 2,417) 29.0 -> 28.9 ms; 158k-cell PISO (135, 1,009) 7.97 -> 8.18 ms.
constexpr int kTailClusterEntries = 2048;
constexpr int kTailBlocks = 8;  // a cluster per vector
constexpr int kTailLanes = 8;   // lanes of a row; lane l hands the row's value to block l
static_assert(kTailLanes == kTailBlocks, "a lane per block");
constexpr int kTailRows = kTailThreads / kTailLanes;
static_assert(kTailMax <= kTailBlocks * kTailRows && kDenseMax <= kTailRows, "one row per group of lanes");

struct TailLevel
{
    int n, nc, nnz;  // nnz: most entries in one block's rows
    const int *rs, *cols, *agg, *ms, *mem;
    const float *val, *dinv, *dense;
    const float* b;  // this level's right-hand side and output: a vector's
    float* o;        // values `stride` apart, vector q at offset q
    int stride;
    float scale;     // coarse-correction scaling
    Sweeps w;
};

/// block `rank`'s share of n rows begins at
__host__ __device__ constexpr int tailFirst(int n, int rank) { return n * rank / kTailBlocks; }
/// the most rows of one share
__host__ __device__ constexpr int tailShare(int n) { return (n + kTailBlocks - 1) / kTailBlocks; }

/// Shared-memory layout of a k_amg_tail block (4-byte words).  Its share of
/// the level's CSR (rs, cols, val) and of the dense inverse's rows; whole:
/// dinv, agg and the aggregates' member lists (ms nc + 1, mem n), the vectors
/// b, x, r (n each), bc and xc (nc each).
__host__ __device__ constexpr size_t tailSmemWords(int n, int nnz, int nc)
{
    return static_cast<size_t>(tailShare(n) + 1) + 2 * static_cast<size_t>(nnz) +
           static_cast<size_t>(tailShare(nc)) * static_cast<size_t>(nc) + 6 * static_cast<size_t>(n) +
           static_cast<size_t>(nc + 1) + 2 * static_cast<size_t>(nc);
}

/// An asynchronous copy of one word to shared address `to`.
__device__ __forceinline__ void copyWord(unsigned to, const void* from)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(from) : "memory");
}
/// v at p of block `block` of the cluster
__device__ __forceinline__ void putAt(float* p, int block, float v)
{
    unsigned at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(block));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

/// The last aggregation level (at most kTailMax rows) and the coarsest solve
/// as one cluster per vector: the sweeps and the residual, restriction, dense
/// solve, prolongation and the sweeps again.  Every block holds the vectors
/// whole and an eighth of the rows of the level and of the dense inverse; the
/// eight lanes that sum a row hand its value to the eight blocks, and a
/// cluster barrier ends each product.  In one block the products were its
/// 11 us: some 20k entries of three shared-memory words each, read with the
/// conflicts of ragged rows.  Cluster q works on vector q and does nothing
/// when done[q] is set (done may be null).
__global__ void __launch_bounds__(kTailThreads) __cluster_dims__(kTailBlocks, 1, 1)
k_amg_tail(const int* done, TailLevel T)
{
    pdl_entry();
    const int q = blockIdx.x / kTailBlocks, rank = blockIdx.x % kTailBlocks;
    if (done && done[q]) return;
    clusterArrive();  // waited for before the first value goes to another block
    extern __shared__ __align__(16) int tsm[];
    const int n = T.n, nc = T.nc, t = threadIdx.x;
    const int lo = tailFirst(n, rank), rows = tailFirst(n, rank + 1) - lo;
    const int lod = tailFirst(nc, rank), rowsd = tailFirst(nc, rank + 1) - lod;
    int* rs = tsm;
    int* cols = rs + tailShare(n) + 1;
    float* val = reinterpret_cast<float*>(cols + T.nnz);
    float* dense = val + T.nnz;
    float* dinv = dense + tailShare(nc) * nc;
    int* agg = reinterpret_cast<int*>(dinv + n);
    int* mem = agg + n;
    int* ms = mem + n;
    float* b = reinterpret_cast<float*>(ms + nc + 1);
    float* x = b + n;
    float* r = x + n;
    float* bc = r + n;
    float* xc = bc + nc;
    // every copy is under way before the first is waited for
    auto copy = [&](void* to, const void* from, int words) {
        const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(to));
        for (int i = t; i < words; i += kTailThreads) copyWord(at + 4u * static_cast<unsigned>(i), static_cast<const int*>(from) + i);
    };
    const int e0 = T.rs[lo], entries = T.rs[lo + rows] - e0;
    copy(dinv, T.dinv, n);
    copy(agg, T.agg, n);
    copy(mem, T.mem, n);
    copy(ms, T.ms, nc + 1);
    copy(rs, T.rs + lo, rows + 1);
    copy(dense, T.dense + static_cast<size_t>(lod) * nc, rowsd * nc);
    for (int i = t; i < n; i += kTailThreads)
        copyWord(static_cast<unsigned>(__cvta_generic_to_shared(b + i)), T.b + static_cast<size_t>(i) * T.stride + q);
    copy(val, T.val + e0, entries);
    copy(cols, T.cols + e0, entries);
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int i = t; i < n; i += kTailThreads) x[i] = T.w.w[0] * dinv[i] * b[i];  // its own copies
    __syncthreads();
    clusterWait();
    const int l = t % kTailLanes, mine = t / kTailLanes;  // the group's row of the share, its aggregate
    // every lane: (A v) of the group's row
    auto product = [&](const float* v) {
        float s = 0.0f;
        if (mine < rows)
            for (int e = rs[mine] - e0 + l; e < rs[mine + 1] - e0; e += kTailLanes) s += val[e] * v[cols[e]];
#pragma unroll
        for (int o = kTailLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    const int i = lo + mine;  // the group's row
    // out = f((A in)_i) in every block
    auto pass = [&](const float* in, float* out, auto f) {
        const float s = product(in);
        if (mine < rows) putAt(out + i, l, f(s));
        clusterArrive();
        clusterWait();
    };
    float *u = x, *v = r;
    auto sweep = [&](float w) {
        pass(u, v, [&](float s) { return u[i] + w * dinv[i] * (b[i] - s); });
        float* const c = u;
        u = v;
        v = c;
    };
    for (int k = 1; k < T.w.m; ++k) sweep(T.w.w[k]);
    pass(u, v, [&](float s) { return b[i] - s; });
    // restriction, in every block
    {
        float s = 0.0f;
        if (mine < nc)
            for (int k = ms[mine] + l; k < ms[mine + 1]; k += kTailLanes) s += v[mem[k]];
#pragma unroll
        for (int o = kTailLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (mine < nc && l == 0) bc[mine] = s;
    }
    __syncthreads();
    // the coarsest solve xc = M bc: a warp per row of the share
    {
        const int lane = t & 31;
        for (int d = t >> 5; d < rowsd; d += kTailThreads / 32)
        {
            float s = 0.0f;
            for (int j = lane; j < nc; j += 32) s += dense[d * nc + j] * bc[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane < kTailBlocks) putAt(xc + lod + d, lane, s);
        }
    }
    clusterArrive();
    clusterWait();
    for (int k = t; k < n; k += kTailThreads) u[k] = u[k] + T.scale * xc[agg[k]];
    __syncthreads();
    for (int k = T.w.m - 1; k > 0; --k) sweep(T.w.w[k]);
    const float s = product(u);
    if (mine < rows && l == 0) T.o[static_cast<size_t>(i) * T.stride + q] = u[i] + T.w.w[0] * dinv[i] * (b[i] - s);
}

constexpr int kTailBlockLanes = 4;

/// Shared-memory layout of k_amg_tail_block (4-byte words): the level's CSR
/// (rs n + 1, cols nnz, val nnz), dinv n, agg n, the aggregates' member
/// lists (ms nc + 1, mem n), the dense inverse nc * nc, the vectors b, x, r
/// n each, bc and xc nc each.
__host__ __device__ constexpr size_t tailBlockWords(int n, int nnz, int nc)
{
    return static_cast<size_t>(n + 1) + 2 * static_cast<size_t>(nnz) + 2 * static_cast<size_t>(n) +
           static_cast<size_t>(nc + 1) + static_cast<size_t>(n) + static_cast<size_t>(nc) * nc + 3 * static_cast<size_t>(n) +
           2 * static_cast<size_t>(nc);
}

/// The same for a small level (kTailClusterEntries): the last aggregation
/// level and the coarsest solve in one block per vector, the level held in shared memory: one coalesced
/// load of its matrix, aggregates, dense inverse and right-hand side, then
/// the sweeps and the residual, restriction, dense solve, prolongation and
/// the sweeps again, separated by block barriers.  Block q works on vector q
/// and does nothing when done[q] is set (done may be null); only the output
/// goes back to global memory.
__global__ void __launch_bounds__(kTailThreads) k_amg_tail_block(const int* done, TailLevel T)
{
    pdl_entry();
    const int q = blockIdx.x;
    if (done && done[q]) return;
    extern __shared__ __align__(16) int tsm[];
    const int n = T.n, nc = T.nc, nnz = T.nnz, t = threadIdx.x;
    int* rs = tsm;
    int* cols = rs + (n + 1);
    float* val = reinterpret_cast<float*>(cols + nnz);
    float* dinv = val + nnz;
    int* agg = reinterpret_cast<int*>(dinv + n);
    int* ms = agg + n;
    int* mem = ms + (nc + 1);
    float* dense = reinterpret_cast<float*>(mem + n);
    float* b = dense + static_cast<size_t>(nc) * nc;
    float* x = b + n;
    float* r = x + n;
    float* bc = r + n;
    float* xc = bc + nc;
    for (int i = t; i <= n; i += kTailThreads) rs[i] = T.rs[i];
    for (int e = t; e < nnz; e += kTailThreads)
    {
        cols[e] = T.cols[e];
        val[e] = T.val[e];
    }
    for (int i = t; i < n; i += kTailThreads)
    {
        const float di = T.dinv[i], bi = T.b[static_cast<size_t>(i) * T.stride + q];
        dinv[i] = di;
        agg[i] = T.agg[i];
        mem[i] = T.mem[i];
        b[i] = bi;
        x[i] = T.w.w[0] * di * bi;
    }
    for (int i = t; i <= nc; i += kTailThreads) ms[i] = T.ms[i];
    for (int i = t; i < nc * nc; i += kTailThreads) dense[i] = T.dense[i];
    __syncthreads();
    const int l = t % kTailBlockLanes, first = t / kTailBlockLanes, stride = kTailThreads / kTailBlockLanes;
    // out(i, (A v)_i) for every row, a group of lanes per row
    auto product = [&](const float* v, auto out) {
        for (int i0 = first;; i0 += stride)
        {
            const int base = i0 - (t % 32) / kTailBlockLanes;
            if (base >= n) break;
            const int i = i0 < n ? i0 : -1;
            float s = 0.0f;
            if (i >= 0)
                for (int e = rs[i] + l; e < rs[i + 1]; e += kTailBlockLanes) s += val[e] * v[cols[e]];
#pragma unroll
            for (int o = kTailBlockLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (i >= 0 && l == 0) out(i, s);
        }
        __syncthreads();
    };
    float *u = x, *v = r;
    for (int k = 1; k < T.w.m; ++k)
    {
        const float w = T.w.w[k];
        product(u, [&](int i, float s) { v[i] = u[i] + w * dinv[i] * (b[i] - s); });
        float* const c = u;
        u = v;
        v = c;
    }
    product(u, [&](int i, float s) { v[i] = b[i] - s; });
    // restriction
    for (int I0 = first;; I0 += stride)
    {
        const int base = I0 - (t % 32) / kTailBlockLanes;
        if (base >= nc) break;
        const int I = I0 < nc ? I0 : -1;
        float s = 0.0f;
        if (I >= 0)
            for (int k = ms[I] + l; k < ms[I + 1]; k += kTailBlockLanes) s += v[mem[k]];
#pragma unroll
        for (int o = kTailBlockLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (I >= 0 && l == 0) bc[I] = s;
    }
    __syncthreads();
    // the coarsest solve xc = M bc, a warp per row
    {
        const int lane = t & 31;
        for (int i = t >> 5; i < nc; i += kTailThreads / 32)
        {
            float s = 0.0f;
            for (int j = lane; j < nc; j += 32) s += dense[i * nc + j] * bc[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) xc[i] = s;
        }
    }
    __syncthreads();
    for (int i = t; i < n; i += kTailThreads) u[i] = u[i] + T.scale * xc[agg[i]];
    __syncthreads();
    for (int k = T.w.m - 1; k > 0; --k)
    {
        const float w = T.w.w[k];
        product(u, [&](int i, float s) { v[i] = u[i] + w * dinv[i] * (b[i] - s); });
        float* const c = u;
        u = v;
        v = c;
    }
    const float w = T.w.w[0];
    product(u, [&](int i, float s) {
        T.o[static_cast<size_t>(i) * T.stride + q] = u[i] + w * dinv[i] * (b[i] - s);
    });
}

/// the coarsest solve x = M b with the dense inverse, when the tail kernel
/// does not hold the level above it (block q: vector q)
__global__ void __launch_bounds__(kDenseMax) k_amg_dense(const int* done, int n, int stride,
                                                         const float* __restrict__ m, const float* b,
                                                         float* __restrict__ x)
{
    pdl_entry();
    const int q = blockIdx.x;
    if (done && done[q]) return;
    const int i = threadIdx.x;
    if (i >= n) return;
    float s = 0.0f;
    for (int j = 0; j < n; ++j) s += m[i * n + j] * b[j * stride + q];
    x[i * stride + q] = s;
}

/// a host CSR pattern whose entries remember where their values live
struct Pattern
{
    int n = 0;
    std::vector<int> rs, cols, pos;
};

/// aggregation (the two phases of the file comment) over the entries that
/// `link` marks (null: every entry, plain aggregation); a row's own diagonal
/// entry always counts
int aggregate(const Pattern& A, std::vector<int>& agg, const std::vector<char>* link = nullptr)
{
    auto on = [&](int e) { return !link || (*link)[static_cast<size_t>(e)]; };
    agg.assign(static_cast<size_t>(A.n), -1);
    int na = 0;
    for (int i = 0; i < A.n; ++i)
    {
        if (agg[i] >= 0) continue;
        bool free = true;
        for (int e = A.rs[i]; e < A.rs[i + 1] && free; ++e)
            if (on(e)) free = agg[A.cols[e]] < 0;
        if (!free) continue;
        for (int e = A.rs[i]; e < A.rs[i + 1]; ++e)
            if (on(e)) agg[A.cols[e]] = na;
        agg[i] = na++;
    }
    for (int i = 0; i < A.n; ++i)
    {
        if (agg[i] >= 0) continue;
        for (int e = A.rs[i]; e < A.rs[i + 1]; ++e)
            if (on(e) && agg[A.cols[e]] >= 0 && A.cols[e] != i)
            {
                agg[i] = agg[A.cols[e]];
                break;
            }
        if (agg[i] < 0) agg[i] = na++;
    }
    return na;
}

/// The strong entries of a level for strength-of-connection aggregation:
/// entry (i, j), j != i, is strong when |a_ij| >= theta * max over k != i of
/// |a_ik| (values indexed by the pattern's positions); diagonal entries are
/// marked too.  Aggregating over strong entries only lines the aggregates
/// up with the strongly coupled directions of an anisotropic operator
/// (cells much thinner across the channel than along it), where plain
/// aggregation mixes weak and strong couplings and the V-cycle loses its
/// contraction.
std::vector<char> strongEntries(const Pattern& A, const std::vector<double>& v, double theta)
{
    std::vector<char> link(A.cols.size(), 0);
    for (int i = 0; i < A.n; ++i)
    {
        double mx = 0.0;
        for (int e = A.rs[i]; e < A.rs[i + 1]; ++e)
            if (A.cols[e] != i) mx = std::max(mx, std::abs(v[static_cast<size_t>(A.pos[e])]));
        for (int e = A.rs[i]; e < A.rs[i + 1]; ++e)
            link[static_cast<size_t>(e)] = A.cols[e] == i || std::abs(v[static_cast<size_t>(A.pos[e])]) >= theta * mx;
    }
    return link;
}

/// Whether the couplings that are not strong are hardly any: at least a tenth
/// of the entries, and on average below kDecoupled of their rows' largest.
/// The aggregates then never join across them, what the V-cycle leaves lies in
/// their direction, and more sweeps on the coarse levels do not reach it.
/// Poisson solves with theta 0.25 on channels of 266k and 689k cells that are
/// long by 2.5, 5, 10 and 20 (mean weak coupling 0.16, 0.04, 0.01, 0.0025), ms
/// with single / weighted sweeps: 4.3 / 4.0 and 7.9 / 6.1, 7.2 / 6.7 and 14.6 /
/// 11.1, 12.6 / 14.0 and 22.0 / 20.2, 8.1 / 11.0 and 15.4 / 17.8.
constexpr double kDecoupled = 0.02;
bool decoupled(const Pattern& A, const std::vector<double>& v, const std::vector<char>& strong)
{
    double sum = 0.0;
    size_t weak = 0;
    for (int i = 0; i < A.n; ++i)
    {
        double mx = 0.0, s = 0.0;
        for (int e = A.rs[i]; e < A.rs[i + 1]; ++e)
        {
            const double a = std::abs(v[static_cast<size_t>(A.pos[e])]);
            if (A.cols[e] != i) mx = std::max(mx, a);
            if (strong[static_cast<size_t>(e)]) continue;
            s += a;
            ++weak;
        }
        if (s > 0.0) sum += s / mx;
    }
    return 10 * weak >= A.cols.size() && sum < kDecoupled * static_cast<double>(weak);
}

}  // namespace

/// A hierarchy's structure from the device matrix pattern (and, for
/// strength of connection, the operator's values).
void Ctx::amgSetup(AmgUse use, const double* vals, double theta)
{
    const auto t0 = std::chrono::steady_clock::now();
    std::unique_ptr<AmgState> a(new AmgState());
    a->theta = theta;
    const int n0 = dm_.nC;
    // the finest pattern from the SELL slices, entries in row order
    Pattern P;
    {
        std::vector<int> start(static_cast<size_t>(nSlices_) + 1), col(static_cast<size_t>(nSlicesEntries_));
        CFG_CUDA(cudaMemcpyAsync(start.data(), dm_.mStart, start.size() * sizeof(int), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaMemcpyAsync(col.data(), dm_.mCol, col.size() * sizeof(int), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
        P.n = n0;
        P.rs.assign(static_cast<size_t>(n0) + 1, 0);
        for (int c = 0; c < n0; ++c)
        {
            const int sl = c >> 5, lane = c & 31;
            for (int e = start[sl] + lane; e < start[sl + 1]; e += 32)
            {
                if (col[e] < 0) break;
                P.cols.push_back(col[e]);
                P.pos.push_back(e);
            }
            P.rs[c + 1] = static_cast<int>(P.cols.size());
        }
    }
    // strength of connection needs the operator's values on every level: the
    // finest from the device (indexed by SELL position), the coarser ones as
    // FP64 Galerkin sums on the host, in the order the device sums them
    std::vector<double> v;
    if (theta > 0)
    {
        if (!vals) fail(CFG_EINVAL, "amg: strength-of-connection aggregation needs the operator's values");
        v.resize(static_cast<size_t>(nSlicesEntries_));
        CFG_CUDA(cudaMemcpyAsync(v.data(), vals, v.size() * sizeof(double), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
    }
    while (true)
    {
        AmgLevel L;
        L.n = P.n;
        // the finest level always aggregates (it reads FP64 in and out)
        if (P.n <= kDenseMax && !a->lv.empty())
        {
            a->nc = P.n;
            a->hrs = P.rs;
            a->hcols = P.cols;
            L.b = alloc<float>(P.n);
            L.x = alloc<float>(P.n);
            a->lv.push_back(L);
            break;
        }
        std::vector<int> agg;
        int na = -1;
        if (theta > 0)
        {
            // a level that the strong entries coarsen by less than half is
            // aggregated plainly instead
            const std::vector<char> link = strongEntries(P, v, theta);
            if (a->lv.empty()) a->decoupled = decoupled(P, v, link);
            na = aggregate(P, agg, &link);
            if (na > P.n / 2) na = -1;
        }
        if (na < 0) na = aggregate(P, agg);
        if (na > P.n * 9 / 10 || na > 0x3fffffff)
            fail(CFG_ESETUP, "amg: the aggregation stopped coarsening above " + std::to_string(kDenseMax) + " rows");
        // members of each aggregate, in row order
        std::vector<int> ms(static_cast<size_t>(na) + 1, 0), mem(static_cast<size_t>(P.n));
        for (int i = 0; i < P.n; ++i) ++ms[agg[i] + 1];
        for (int I = 0; I < na; ++I) ms[I + 1] += ms[I];
        {
            std::vector<int> fill(ms.begin(), ms.end() - 1);
            for (int i = 0; i < P.n; ++i) mem[fill[agg[i]]++] = i;
        }
        // the coarse pattern and, per coarse entry, the fine entries it sums
        Pattern C;
        C.n = na;
        C.rs.assign(static_cast<size_t>(na) + 1, 0);
        std::vector<int> gs{0}, gl;
        std::vector<std::pair<int, int>> row;  // (coarse column, fine entry index)
        for (int I = 0; I < na; ++I)
        {
            row.clear();
            for (int k = ms[I]; k < ms[I + 1]; ++k)
            {
                const int i = mem[k];
                for (int e = P.rs[i]; e < P.rs[i + 1]; ++e) row.push_back({agg[P.cols[e]], e});
            }
            std::stable_sort(row.begin(), row.end(),
                             [](const std::pair<int, int>& x, const std::pair<int, int>& y) { return x.first < y.first; });
            for (size_t k = 0; k < row.size(); ++k)
            {
                if (k == 0 || row[k].first != row[k - 1].first)
                {
                    if (k > 0) gs.push_back(static_cast<int>(gl.size()));
                    C.cols.push_back(row[k].first);
                }
                gl.push_back(P.pos[row[k].second]);
            }
            if (!row.empty()) gs.push_back(static_cast<int>(gl.size()));
            C.rs[I + 1] = static_cast<int>(C.cols.size());
        }
        C.pos.resize(C.cols.size());
        std::iota(C.pos.begin(), C.pos.end(), 0);
        if (theta > 0)
        {
            std::vector<double> vc(C.cols.size());
            for (size_t k = 0; k < vc.size(); ++k)
            {
                double t = 0.0;
                for (int g = gs[k]; g < gs[k + 1]; ++g) t += v[static_cast<size_t>(gl[static_cast<size_t>(g)])];
                vc[k] = t;
            }
            v.swap(vc);
        }
        L.agg = upload(agg);
        L.ms = upload(ms);
        L.mem = upload(mem);
        L.gs = upload(gs);
        L.gl = upload(gl);
        L.nnzNext = static_cast<int>(C.cols.size());
        if (!a->lv.empty())
        {
            std::vector<int> dpos(static_cast<size_t>(P.n), -1);
            for (int i = 0; i < P.n; ++i)
                for (int e = P.rs[i]; e < P.rs[i + 1]; ++e)
                    if (P.cols[e] == i) dpos[i] = e;
            L.rs = upload(P.rs);
            L.cols = upload(P.cols);
            L.dpos = upload(dpos);
            L.val = alloc<float>(P.cols.size());
            if (P.n >= kSellMinRows)
            {
                // SELL-32: slice s holds rows 32s..32s+31, entry k of row r at
                // start[s] + (r & 31) + 32 k, slices as wide as their longest row
                const int nsl = (P.n + 31) / 32;
                std::vector<int> sst(static_cast<size_t>(nsl) + 1, 0);
                for (int sl = 0; sl < nsl; ++sl)
                {
                    int w = 0;
                    for (int r = sl * 32; r < std::min(P.n, sl * 32 + 32); ++r) w = std::max(w, P.rs[r + 1] - P.rs[r]);
                    sst[static_cast<size_t>(sl) + 1] = sst[static_cast<size_t>(sl)] + 32 * w;
                }
                std::vector<int> scol(static_cast<size_t>(sst[static_cast<size_t>(nsl)]), -1), pos(P.cols.size());
                for (int r = 0; r < P.n; ++r)
                    for (int e = P.rs[r]; e < P.rs[r + 1]; ++e)
                    {
                        const int p = sst[static_cast<size_t>(r >> 5)] + (r & 31) + 32 * (e - P.rs[r]);
                        scol[static_cast<size_t>(p)] = P.cols[e];
                        pos[static_cast<size_t>(e)] = p;
                    }
                L.sstart = upload(sst);
                L.scol = upload(scol);
                L.sellPos = upload(pos);
                L.sval = alloc<float>(std::max<size_t>(scol.size(), 1));
                CFG_CUDA(cudaMemsetAsync(L.sval, 0, std::max<size_t>(scol.size(), 1) * sizeof(float), stream_));
            }
        }
        L.dinv = alloc<float>(P.n);
        L.b = alloc<float>(P.n);
        L.x = alloc<float>(P.n);
        L.r = alloc<float>(P.n);
        L.xo = alloc<float>(P.n);
        a->lv.push_back(L);
        P = std::move(C);
    }
    // the coarsest level's CSR operator (for the Galerkin values and its inverse)
    {
        AmgLevel& L = a->lv.back();
        L.val = alloc<float>(std::max<size_t>(P.cols.size(), 1));
        a->dense = alloc<float>(static_cast<size_t>(P.n) * P.n);
    }
    // lane groups: about two entries (or aggregate members) per lane, at
    // least four lanes, and fewer while the level's rows times the group
    // would need more than one wave of resident threads
    {
        const double resident = static_cast<double>(sms_) * 2048;
        auto pick = [&](double avg, int count) {
            int g = 4;
            while (g < 32 && g < avg / 2.0) g *= 2;
            while (g > 4 && static_cast<double>(count) * g > resident) g /= 2;
            return g;
        };
        for (size_t l = 0; l + 1 < a->lv.size(); ++l)
        {
            AmgLevel& V = a->lv[l];
            const AmgLevel& N = a->lv[l + 1];
            V.gAgg = pick(static_cast<double>(V.n) / N.n, N.n);
            if (l >= 1) V.gRow = pick(static_cast<double>(a->lv[l - 1].nnzNext) / V.n, V.n);
        }
    }
    // the tail level's shared-memory copy, when a block's part fits in its
    // opt-in shared memory (set before any stream capture)
    if (const int T = static_cast<int>(a->lv.size()) - 2; T >= 1 && a->lv[static_cast<size_t>(T)].n <= kTailMax)
    {
        const int n = a->lv[static_cast<size_t>(T)].n;
        std::vector<int> rs(static_cast<size_t>(n) + 1);
        CFG_CUDA(cudaMemcpyAsync(rs.data(), a->lv[static_cast<size_t>(T)].rs, rs.size() * sizeof(int), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
        int nnz = 0;
        for (int k = 0; k < kTailBlocks; ++k)
            nnz = std::max(nnz, rs[static_cast<size_t>(tailFirst(n, k + 1))] - rs[static_cast<size_t>(tailFirst(n, k))]);
        const int nc = a->lv[static_cast<size_t>(T) + 1].n, all = rs[static_cast<size_t>(n)];
        a->tailCluster = all > kTailClusterEntries && clusterMax_ >= kTailBlocks;
        if (!a->tailCluster) nnz = all;
        const size_t bytes = 4 * (a->tailCluster ? tailSmemWords(n, nnz, nc) : tailBlockWords(n, nnz, nc));
        int optin = 0;
        CFG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device_));
        if (bytes <= static_cast<size_t>(optin))
        {
            // the attribute belongs to the kernel on this device, which every
            // hierarchy of every context shares: it only ever grows
            static std::mutex mu;
            static std::vector<std::pair<int, size_t>> granted;  // (device, bytes)
            std::lock_guard<std::mutex> lock(mu);
            auto it = std::find_if(granted.begin(), granted.end(),
                                   [&](const std::pair<int, size_t>& g) { return g.first == device_; });
            if (it == granted.end() || it->second < bytes)
            {
                for (const auto kernel : {k_amg_tail, k_amg_tail_block})
                    CFG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
                if (it == granted.end()) granted.push_back({device_, bytes});
                else it->second = bytes;
            }
            a->tailSmem = bytes;
            a->tailNnz = nnz;
        }
    }
    CFG_CUDA(cudaStreamSynchronize(stream_));
    a->setupMs = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    amgSlot(use).reset(a.release());
}

/// The hierarchy's values from the finest operator (FP64 SELL values and
/// diagonal): Galerkin sums level by level, inverse diagonals, and the
/// coarsest level's dense inverse (on the host).
void Ctx::amgValues(AmgUse use, const double* vals, const double* diag, const float* vals32)
{
    auto& slot = amgSlot(use);
    if (!slot) amgSetup(use, vals, use == kAmgPressure ? amgTheta_ : 0.0);
    AmgState& a = *slot;
    const auto t0 = std::chrono::steady_clock::now();
    a.vals32 = vals32;
    k_amg_dinv0<<<GS_, TPB, 0, stream_>>>(dm_.nC, diag, a.lv[0].dinv);
    for (size_t l = 0; l + 1 < a.lv.size(); ++l)
    {
        const AmgLevel& L = a.lv[l];
        AmgLevel& N = a.lv[l + 1];
        const int g = std::max(1, std::min((L.nnzNext + TPB - 1) / TPB, sms_ * 8));
        k_amg_galerkin<<<g, TPB, 0, stream_>>>(L.nnzNext, L.gs, L.gl, l == 0 ? vals : nullptr, l == 0 ? nullptr : L.val,
                                               N.val);
        if (N.sstart) k_amg_to_sell<<<g, TPB, 0, stream_>>>(L.nnzNext, N.sellPos, N.val, N.sval);
        if (l + 2 < a.lv.size())
            k_amg_dinv<<<std::max(1, std::min((N.n + TPB - 1) / TPB, sms_ * 8)), TPB, 0, stream_>>>(N.n, N.dpos, N.val,
                                                                                                N.dinv);
        launchCheck("amg_galerkin", 2);
    }
    // dense inverse of the coarsest operator, Gauss-Jordan with partial
    // pivoting; a singular operator (pure Neumann) gets a small diagonal shift
    {
        const int n = a.nc;
        std::vector<float> v(a.hcols.size());
        double theta = 0.0;
        if (use == kAmgMomentum)
        {
            if (!a.skew) a.skew = alloc<double>(1);
            CFG_CUDA(cudaMemsetAsync(a.skew, 0, sizeof(double), stream_));
            k_amg_skew<<<GS_, TPB, 0, stream_>>>(DMat{dm_.nC, dm_.mStart, dm_.mCol}, vals,
                                                 reinterpret_cast<unsigned long long*>(a.skew));
            launchCheck("amg_skew");
            CFG_CUDA(cudaMemcpyAsync(&theta, a.skew, sizeof(double), cudaMemcpyDeviceToHost, stream_));
        }
        if (!v.empty())
            CFG_CUDA(cudaMemcpyAsync(v.data(), a.lv.back().val, v.size() * sizeof(float), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
        a.skewClass = skewOf(theta);
        std::vector<double> m(static_cast<size_t>(n) * n, 0.0), inv(static_cast<size_t>(n) * n, 0.0);
        double dmax = 0;
        for (int i = 0; i < n; ++i)
            for (int e = a.hrs[i]; e < a.hrs[i + 1]; ++e)
            {
                m[static_cast<size_t>(i) * n + a.hcols[e]] += v[e];
                if (a.hcols[e] == i) dmax = std::max(dmax, std::abs(static_cast<double>(v[e])));
            }
        for (int i = 0; i < n; ++i)
        {
            m[static_cast<size_t>(i) * n + i] += 1e-6 * dmax;
            inv[static_cast<size_t>(i) * n + i] = 1.0;
        }
        for (int c = 0; c < n; ++c)
        {
            int piv = c;
            for (int i = c + 1; i < n; ++i)
                if (std::abs(m[static_cast<size_t>(i) * n + c]) > std::abs(m[static_cast<size_t>(piv) * n + c])) piv = i;
            if (piv != c)
                for (int j = 0; j < n; ++j)
                {
                    std::swap(m[static_cast<size_t>(c) * n + j], m[static_cast<size_t>(piv) * n + j]);
                    std::swap(inv[static_cast<size_t>(c) * n + j], inv[static_cast<size_t>(piv) * n + j]);
                }
            const double d = m[static_cast<size_t>(c) * n + c];
            if (!(std::abs(d) > 0)) fail(CFG_ENUMERIC, "amg: singular coarsest operator");
            for (int j = 0; j < n; ++j)
            {
                m[static_cast<size_t>(c) * n + j] /= d;
                inv[static_cast<size_t>(c) * n + j] /= d;
            }
            for (int i = 0; i < n; ++i)
            {
                if (i == c) continue;
                const double f = m[static_cast<size_t>(i) * n + c];
                if (f == 0) continue;
                for (int j = 0; j < n; ++j)
                {
                    m[static_cast<size_t>(i) * n + j] -= f * m[static_cast<size_t>(c) * n + j];
                    inv[static_cast<size_t>(i) * n + j] -= f * inv[static_cast<size_t>(c) * n + j];
                }
            }
        }
        std::vector<float> invf(inv.begin(), inv.end());
        if (!invf.empty())
            CFG_CUDA(cudaMemcpyAsync(a.dense, invf.data(), invf.size() * sizeof(float), cudaMemcpyHostToDevice, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
    }
    a.valuesReady = true;
    a.valuesMs = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

/// z = V-cycle(r), r and z in FP64 on device cells.  Inside the device FCG
/// every kernel stops once the solve is done (st->done) and the finest
/// post-smoothing also forms z.q and beta.
void Ctx::amgApply(const double* r, double* z)
{
    amgCycle(r, z, nullptr, nullptr, kSingleSweeps);
}

namespace
{
template <class V>
V* vecOf(float* one, float* three);
template <>
float* vecOf<float>(float* one, float*)
{
    return one;
}
template <>
float4* vecOf<float4>(float*, float* three)
{
    return reinterpret_cast<float4*>(three);
}

template <class V>
Coarse<V> coarseOf(const AmgLevel& L)
{
    Coarse<V> c{};
    c.n = L.n;
    c.rs = L.rs;
    c.cols = L.cols;
    c.val = L.val;
    c.dinv = L.dinv;
    c.agg = L.agg;
    c.ms = L.ms;
    c.mem = L.mem;
    c.sstart = L.sstart;
    c.scol = L.scol;
    c.sval = L.sval;
    c.b = vecOf<V>(L.b, L.b3);
    c.x = vecOf<V>(L.x, L.x3);
    c.r = vecOf<V>(L.r, L.r3);
    c.o = vecOf<V>(L.xo, L.xo3);
    c.gRow = L.gRow;
    c.gAgg = L.gAgg;
    return c;
}

/// The sweeps of the coarse levels in the solvers' V-cycles.  The plain
/// aggregation hierarchy loses its contraction on the coarse levels, where
/// sweeps cost a fraction of the finest level's; as Chebyshev polynomials over
/// [lo, 1.9] (D^-1 A reaches 2 at most) two to four of them go further than
/// damped Jacobi.  On the 2M-cell channel (B200, one outer iteration to
/// 1e-12): one sweep 301 ms (1182 momentum component-iterations, 206 pressure
/// iterations), two 178 ms (595, 131), three 170 ms (533, 101), four on the
/// first coarse level and two below 159 ms (471, 106).  Two take the 158k-cell
/// PISO step from 10.6 to 8.6 ms, four to 9.7.  Three pay from kSellMinRows
/// rows on, where a sweep is not a launch's latency, and four from kFourMinRows
/// on (one outer iteration of channels whose cells are long by 1 to 20, gain
/// over single sweeps in the mean with two / three / four: 282k cells, 36k rows,
/// 1.19 / 1.18 / 1.10 and in the worst case 1.04 / 0.99 / 0.91, the 262k-cell
/// channel of cells long by 2.5 44 -> 33 / 30 / 30 ms; 689k cells, 82k rows, 1.29
/// / 1.31 / 1.25; 1.2M cells, 144k rows, 1.34 / 1.38 / 1.38; 2.1M cells, 250k
/// rows, 1.48 / 1.54 / 1.57).  lo: 0.2 for two sweeps and 0.1 for more;
/// convection narrows the choice (BiCGStab iterations of a
/// numpy model, one sweep / four with lo 0.1 / with lo 0.3 / two damped
/// Jacobi: theta 0.42 45/25/29/37, 0.71 63/57/49/61, 0.83 87/none/70/87, 0.88
/// 110/none/90/107): class 1 takes lo 0.3, and only on large levels, where
/// that is a gain over the launches it adds; class 2 keeps single sweeps.  Its
/// line at theta 0.7, on the GPU (two outer iterations to 1e-10, class 1 /
/// single sweeps): 320k cells theta 0.65-0.71 85 / 91 ms, 0.74-0.78 105 / 114,
/// 0.79-0.82 122 / 128, 0.85-0.87 261 / 144 (1575 / 1337 iterations); 292k
/// cubes 0.63-0.66 69 / 72, 0.70-0.72 77 / 74, 0.78-0.79 83 / 82.
Smoother smootherOf(const AmgState& a, int skewClass)
{
    const int rows = a.lv.size() > 1 ? a.lv[1].n : 0;
    if (skewClass == kSingleSweeps || (skewClass == 1 && rows < kSellMinRows)) return singleSweeps();
    const double lo2 = skewClass == 1 ? 0.3 : 0.2, lo4 = skewClass == 1 ? 0.3 : 0.1;
    const Sweeps two = chebyshev(2, lo2, 1.9);
    if (rows < kSellMinRows) return Smoother{two, two};
    return Smoother{chebyshev(skewClass == 1 || rows >= kFourMinRows ? 4 : 3, lo4, 1.9), two};
}

/// The level of the fused tail kernel (the last aggregated level, when it is
/// not the finest and fits), or the dense level.
int lastLevel(const AmgState& a)
{
    const int L = static_cast<int>(a.lv.size());
    return a.tailSmem ? L - 2 : L - 1;
}

/// Everything of a V-cycle below the finest level: from the finest residual
/// (level 0's r) to the finest level's corrected iterate (level 0's r, which
/// the post-sweep reads).
template <class V>
void coarseCycle(const AmgState& a, bool pdl, int sms, cudaStream_t stream, const int* stop, float scale, const Smoother& sm)
{
    constexpr int vectors = sizeof(V) == sizeof(float) ? 1 : 3, stride = sizeof(V) / sizeof(float);
    const int L = static_cast<int>(a.lv.size()), last = lastLevel(a);
    auto grid = [&](int n) { return std::max(1, std::min((n + TPB - 1) / TPB, sms * 8)); };
    // a group of G lanes per coarse row or aggregate
    auto ggrid = [&](int n, int G) { return std::max(1, std::min((n + TPB / G - 1) / (TPB / G), sms * 8)); };
    auto residual = [&](const Coarse<V>& C, const V* x, V* r) {
        if (C.sstart)
            launchK(pdl, k_amg_residual_sell<V>, waveGrid(reinterpret_cast<const void*>(k_amg_residual_sell<V>), sms, C.n),
                    TPB, 0, stream, stop, C, x, r);
        else
            withGroup(C.gRow, [&](auto Gc) {
                constexpr int G = decltype(Gc)::value;
                launchK(pdl, k_amg_residual<V, G>, ggrid(C.n, G), TPB, 0, stream, stop, C, x, r);
            });
    };
    auto smooth = [&](const Coarse<V>& C, float w, const V* y, V* out) {
        if (C.sstart)
            launchK(pdl, k_amg_smooth_sell<V>, waveGrid(reinterpret_cast<const void*>(k_amg_smooth_sell<V>), sms, C.n),
                    TPB, 0, stream, stop, C, w, y, out);
        else
            withGroup(C.gRow, [&](auto Gc) {
                constexpr int G = decltype(Gc)::value;
                launchK(pdl, k_amg_smooth<V, G>, ggrid(C.n, G), TPB, 0, stream, stop, C, w, y, out);
            });
    };
    for (int l = 0; l < last; ++l)
    {
        const Coarse<V> U = coarseOf<V>(a.lv[static_cast<size_t>(l)]), C = coarseOf<V>(a.lv[static_cast<size_t>(l) + 1]);
        const bool inner = l + 1 < last;
        const Sweeps& w = sm.at(l + 1);
        withGroup(U.gAgg, [&](auto Gc) {
            constexpr int G = decltype(Gc)::value;
            launchK(pdl, k_amg_restrict<V, G>, ggrid(C.n, G), TPB, 0, stream, stop, C.n, U.ms, U.mem, U.r,
                    inner ? C.dinv : static_cast<const float*>(nullptr), w.w[0], C.b, C.x);
        });
        if (!inner) break;
        // x, o and r take turns; the iterate ends in x (an odd number of
        // sweeps) or in o
        V *x = C.x, *y = C.o;
        for (int k = 1; k < w.m; ++k)
        {
            smooth(C, w.w[k], x, y);
            std::swap(x, y);
        }
        residual(C, x, C.r);
    }
    const Coarse<V> B = coarseOf<V>(a.lv[static_cast<size_t>(last)]);
    if (a.tailSmem)
    {
        TailLevel t{};
        t.n = B.n;
        t.nc = a.lv[static_cast<size_t>(last) + 1].n;
        t.nnz = a.tailNnz;
        t.rs = B.rs;
        t.cols = B.cols;
        t.agg = B.agg;
        t.ms = B.ms;
        t.mem = B.mem;
        t.val = B.val;
        t.dinv = B.dinv;
        t.dense = a.dense;
        t.b = reinterpret_cast<const float*>(B.b);
        t.o = reinterpret_cast<float*>(B.o);
        t.stride = stride;
        t.scale = scale;
        t.w = sm.at(last);
        if (a.tailCluster) launchK(pdl, k_amg_tail, vectors * kTailBlocks, kTailThreads, a.tailSmem, stream, stop, t);
        else launchK(pdl, k_amg_tail_block, vectors, kTailThreads, a.tailSmem, stream, stop, t);
    }
    else
        launchK(pdl, k_amg_dense, vectors, kDenseMax, 0, stream, stop, a.nc, stride, a.dense,
                reinterpret_cast<const float*>(B.b), reinterpret_cast<float*>(B.x));
    for (int l = last - 1; l >= 0; --l)
    {
        const Coarse<V> C = coarseOf<V>(a.lv[static_cast<size_t>(l)]), N = coarseOf<V>(a.lv[static_cast<size_t>(l) + 1]);
        const Sweeps& w = sm.at(l);
        const bool odd = l == 0 || (w.m & 1);
        V *y = odd ? C.r : C.x, *t = odd ? C.o : C.r;
        launchK(pdl, k_amg_prolong<V>, grid(C.n), TPB, 0, stream, stop, C.n, odd ? C.x : C.o, l + 1 == L - 1 ? N.x : N.o,
                C.agg, y, scale);
        if (l == 0) break;
        // sweeps through the two free vectors in reverse, the last into o
        for (int k = w.m - 1; k > 0; --k)
        {
            smooth(C, w.w[k], y, t);
            std::swap(y, t);
        }
        smooth(C, w.w[0], y, C.o);
    }
}

/// the kernels of coarseCycle
int coarseKernels(const AmgState& a, const Smoother& sm)
{
    int k = 2;
    for (int l = 1; l < lastLevel(a); ++l) k += 2 + 2 * sm.at(l).m;
    return k + 1;
}
}  // namespace

void Ctx::amgCycle(const double* r, double* z, const double* q, FcgState* st, int skewClass, bool swept)
{
    if (!amg_) fail(CFG_EINVAL, "amg: the hierarchy is not set up (amgValues)");
    AmgState& a = *amg_;
    if (!a.valuesReady) fail(CFG_EINVAL, "amg: values not set up");
    const DMat A{dm_.nC, dm_.mStart, dm_.mCol};
    const int* stop = st ? &st->done : nullptr;
    const int Wsel = maxW_ <= 7 ? 7 : (maxW_ <= 16 ? 16 : 0);
    const AmgLevel& V = a.lv[0];
    if (!swept)
    {
        const auto pre0 = Wsel == 7 ? k_amg_pre0<7> : (Wsel == 16 ? k_amg_pre0<16> : k_amg_pre0<0>);
        launchK(amgPdl(), pre0, waveGrid(reinterpret_cast<const void*>(pre0), sms_, A.n), TPB, 0, stream_, stop, A, a.vals32,
                V.dinv, r, V.x, V.r);
    }
    coarseCycle<float>(a, amgPdl(), sms_, stream_, stop, kScale, smootherOf(a, skewClass));
    // one block partial per block: the grid is at most G_ blocks, which
    // partials_ holds
    const auto post0 = Wsel == 7 ? k_amg_post0<7> : (Wsel == 16 ? k_amg_post0<16> : k_amg_post0<0>);
    launchK(amgPdl(), post0, waveGrid(reinterpret_cast<const void*>(post0), sms_, A.n), TPB, 0, stream_, stop, A, a.vals32,
            V.dinv, r, V.r, z, q, partials_, st);
    launchCheck("amg_vcycle", amgCycleKernels(kAmgPressure, skewClass));
}

/// z_q = V-cycle(b_q) for the three components whose done flag is clear
/// (the BiCGStab's flags; a converged component keeps its old z_q)
void Ctx::amgCycle3(AmgUse use, CV3P b, V3P z, const int* done, float scale, int skewClass,
                    const std::function<void(int)>& mark)
{
    if (!amgSlot(use)) fail(CFG_EINVAL, "amg: the hierarchy is not set up (amgValues)");
    AmgState& a = *amgSlot(use);
    if (!a.valuesReady) fail(CFG_EINVAL, "amg: values not set up");
    if (!a.lv[0].x3) fail(CFG_EINVAL, "amg: the three-component vectors are not allocated (amgVectors3)");
    const DMat A{dm_.nC, dm_.mStart, dm_.mCol};
    const int Wsel = maxW_ <= 7 ? 7 : (maxW_ <= 16 ? 16 : 0);
    const AmgLevel& V = a.lv[0];
    float4* const x = reinterpret_cast<float4*>(V.x3);
    float4* const r = reinterpret_cast<float4*>(V.r3);
    const auto pre0 = Wsel == 7 ? k_amgv_pre0<7> : (Wsel == 16 ? k_amgv_pre0<16> : k_amgv_pre0<0>);
    launchK(amgPdl(), pre0, waveGrid(reinterpret_cast<const void*>(pre0), sms_, A.n), TPB, 0, stream_, done, A, a.vals32, V.dinv,
            b, x, r);
    if (mark) mark(0);
    coarseCycle<float4>(a, amgPdl(), sms_, stream_, done, scale, smootherOf(a, skewClass));
    if (mark) mark(1);
    const auto post0 = Wsel == 7 ? k_amgv_post0<7> : (Wsel == 16 ? k_amgv_post0<16> : k_amgv_post0<0>);
    launchK(amgPdl(), post0, waveGrid(reinterpret_cast<const void*>(post0), sms_, A.n), TPB, 0, stream_, done, A, a.vals32,
            V.dinv, b, r, z);
    launchCheck("amg_vcycle3", amgCycleKernels(use, skewClass));
}

/// the class of the momentum operator the hierarchy last took its values from
/// (0 without one), which chooses the sweeps of its V-cycles; the pressure's is 0
int Ctx::amgSkewClass() const { return amgU_ ? amgU_->skewClass : 0; }

void Ctx::setAmgStrength(double theta)
{
    if (!(theta >= 0.0 && theta <= 1.0)) fail(CFG_EINVAL, "amg strength: theta must lie in [0, 1]");
    if (amg_ && amg_->theta != theta)
        fail(CFG_EINVAL, "amg strength: the pressure hierarchy is built already (with theta " +
                             std::to_string(amg_->theta) + "); set the strength before the first AMG pressure solve");
    amgTheta_ = theta;
}

/// The level vectors of the three-component V-cycle, allocated once (before
/// any stream capture that launches amgCycle3).
void Ctx::amgVectors3(AmgUse use)
{
    if (!amgSlot(use)) fail(CFG_EINVAL, "amg: the hierarchy is not set up (amgValues)");
    for (auto& V : amgSlot(use)->lv)
        if (!V.x3)
        {
            const size_t m = 4 * static_cast<size_t>(V.n);  // a float4 per row
            V.b3 = alloc<float>(m);
            V.x3 = alloc<float>(m);
            V.r3 = alloc<float>(m);
            V.xo3 = alloc<float>(m);
        }
}

/// The number of kernels one V-cycle launches.
int Ctx::amgCycleKernels(AmgUse use, int skewClass) const
{
    const AmgState* a = use == kAmgMomentum ? amgU_.get() : amg_.get();
    return a ? 2 + coarseKernels(*a, smootherOf(*a, skewClass)) : 0;
}

namespace
{

/// r = b - A x, |r|2 and |b|2; the solve is done at once when |r|/|b| <= tol
template <int W>
__global__ void __launch_bounds__(TPB) k_fcgd_init(DMat A, const double* __restrict__ val, const double* __restrict__ b,
                                                   const double* __restrict__ x, double* __restrict__ r,
                                                   double* partials, FcgState* st)
{
    const bool inf = st->normType == 0;
    double s[2] = {0.0, 0.0};
    const double* xs[1] = {x};
    FOR_ROWS(c, A.n)
    {
        double y[1];
        spmv_row<W, 1>(A, val, c, xs, y);
        const double bc = b[c], rc = bc - y[0];
        r[c] = rc;
        if (inf)
        {
            s[0] = smax(s[0], fabs(rc));
            s[1] = smax(s[1], fabs(bc));
        }
        else
        {
            s[0] += rc * rc;
            s[1] += bc * bc;
        }
    }
    if (inf) block_max<2>(s);
    else block_sum<2>(s);
    const int G = gridDim.x;
    if (threadIdx.x == 0)
    {
        partials[blockIdx.x] = s[0];
        partials[G + blockIdx.x] = s[1];
    }
    if (!last_block(&st->ticket[0])) return;
    double f[2];
    if (inf) final_max<2>(partials, G, f);
    else final_sum<2>(partials, G, f);
    if (threadIdx.x == 0)
    {
        st->ticket[0] = 0;
        st->it = 0;
        if (inf)
        {
            st->rn = f[0];
            st->bn = smax(f[1], 1e-300);
            st->conv = st->rn / st->bn < st->tol;
        }
        else
        {
            st->rn = sqrt(f[0]);
            st->bn = sqrt(f[1]);
            st->conv = !(st->bn > 0) || st->rn / st->bn <= st->tol;
        }
        st->init = st->rn;
        st->done = st->conv || st->maxIter <= 0;
    }
}

/// q = A p with p.r and p.q; alpha = p.r / p.q, or done on a breakdown.
/// kForm: p = z + beta p is formed here, per column as the row is read (the
/// old p stays for the other rows, the new one goes to pNew); beta is 0 in
/// the first iteration and p zero.
template <int W, bool kForm>
__global__ void __launch_bounds__(TPB) k_fcgd_spmv(DMat A, const double* __restrict__ val, const double* z, const double* p,
                                                   double* __restrict__ pNew, const double* r, double* __restrict__ q,
                                                   double* partials, FcgState* st)
{
    pdl_entry();
    if (st->done) return;
    const double be = st->beta;
    double s[2] = {0.0, 0.0};
    FOR_ROWS(c, A.n)
    {
        double y[1];
        spmv_row_gather<W, 1>(A, val, c, y, [&](int col, double (&xv)[1]) {
            xv[0] = kForm ? z[col] + be * p[col] : p[col];
        });
        q[c] = y[0];
        const double pc = kForm ? z[c] + be * p[c] : p[c];
        if (kForm) pNew[c] = pc;
        s[0] += pc * r[c];
        s[1] += pc * y[0];
    }
    block_sum<2>(s);
    const int G = gridDim.x;
    if (threadIdx.x == 0)
    {
        partials[blockIdx.x] = s[0];
        partials[G + blockIdx.x] = s[1];
    }
    if (!last_block(&st->ticket[0])) return;
    double f[2];
    final_sum<2>(partials, G, f);
    if (threadIdx.x == 0)
    {
        st->ticket[0] = 0;
        if (!(f[1] > 0)) st->done = 1;
        else
        {
            st->pq = f[1];
            st->alpha = f[0] / f[1];
        }
    }
}

/// The end of an update: |r| from the block values in s, and the stopping test
__device__ __forceinline__ void fcg_update_end(double (&s)[1], bool inf, double* partials, FcgState* st)
{
    if (inf) block_max<1>(s);
    else block_sum<1>(s);
    if (threadIdx.x == 0) partials[blockIdx.x] = s[0];
    if (!last_block(&st->ticket[1])) return;
    double f[1];
    if (inf) final_max<1>(partials, gridDim.x, f);
    else final_sum<1>(partials, gridDim.x, f);
    if (threadIdx.x == 0)
    {
        st->ticket[1] = 0;
        st->it = st->it + 1;
        st->rn = inf ? f[0] : sqrt(f[0]);
        if (inf ? st->rn / st->bn < st->tol : st->rn / st->bn <= st->tol)
        {
            st->conv = 1;
            st->done = 1;
        }
        else if (st->it >= st->maxIter || !(st->rn == st->rn))
        {
            st->done = 1;
        }
    }
}

/// x += alpha p, r -= alpha q, |r| and the stopping test
__global__ void __launch_bounds__(TPB) k_fcgd_update(int n, const double* p, const double* q,
                                                     double* __restrict__ x, double* __restrict__ r, double* partials,
                                                     FcgState* st)
{
    pdl_entry();
    if (st->done) return;
    const bool inf = st->normType == 0;
    const double al = st->alpha;
    double s[1] = {0.0};
    FOR_ROWS(c, n)
    {
        x[c] = x[c] + al * p[c];
        const double rc = r[c] - al * q[c];
        r[c] = rc;
        s[0] = inf ? smax(s[0], fabs(rc)) : s[0] + rc * rc;
    }
    fcg_update_end(s, inf, partials, st);
}

/// p = z + beta p
__global__ void __launch_bounds__(TPB) k_fcgd_p(int n, const double* z, double* __restrict__ p,
                                                const FcgState* st)
{
    pdl_entry();
    if (st->done) return;
    const double be = st->beta;
    FOR_ROWS(c, n) p[c] = z[c] + be * p[c];
}

/// x += alpha p, r -= alpha q with |r| and the stopping test, and the
/// V-cycle's finest first sweep and residual of the new r (k_amg_pre0), which
/// is formed per column as the row is read (the old r stays for the other
/// rows).  When the test is met the sweep has been for nothing, once a solve.
template <int W>
__global__ void __launch_bounds__(TPB) k_fcgd_update_pre0(DMat A, const float* __restrict__ val,
                                                          const float* __restrict__ dinv, const double* p, const double* q,
                                                          double* __restrict__ x, const double* r, double* __restrict__ rNew,
                                                          float* __restrict__ xs, float* __restrict__ rs,
                                                          double* partials, FcgState* st)
{
    pdl_entry();
    if (st->done) return;
    const bool inf = st->normType == 0;
    const double al = st->alpha;
    double s[1] = {0.0};
    FOR_ROWS(c, A.n)
    {
        const double rc = r[c] - al * q[c];
        const float sum = sell_row<W>(A, val, c, [&](int j) {
            return kOmega * __ldg(dinv + j) * static_cast<float>(r[j] - al * q[j]);
        });
        const float bc = static_cast<float>(rc);
        x[c] = x[c] + al * p[c];
        rNew[c] = rc;
        xs[c] = kOmega * dinv[c] * bc;
        rs[c] = bc - sum;
        s[0] = inf ? smax(s[0], fabs(rc)) : s[0] + rc * rc;
    }
    fcg_update_end(s, inf, partials, st);
}

/// Up to this many rows the search direction is formed in the product and the
/// update in the first sweep: two launches fewer per iteration for a second
/// gathered vector in each (158k-cell PISO step 9.5 -> 8.4 ms, 55k-tet Poisson
/// 3.27 -> 3.16 ms; above it the gathers cost more than the launches: 262k
/// cells 31.4 -> 31.6 ms, 1.2M 16.4 -> 16.8 ms, 2M 158.7 -> 162.6 ms; Poisson
/// solves of 195k, 216k, 275k and 348k cubes 3.49 -> 3.33, 3.58 -> 3.43, 3.96 ->
/// 3.92 and 4.42 -> 4.47 ms).
constexpr int kFormRows = 200000;

}  // namespace

/// Flexible CG (FCG(1): alpha = p.r / p.q, beta = -z.q / p.q) with the AMG
/// V-cycle as preconditioner, to |b - A x|2 / |b|2 <= tol (normType 1) or
/// the reference's |r|inf test (0), with every scalar on the device: the
/// host polls the state once per chunk of iterations, and each chunk is a
/// CUDA graph captured once.
void Ctx::amgFcg(const double* vals, const double* b, double* x, double tol, int maxIter, int normType,
                 cfg_solver_report* rep)
{
    if (!amg_) fail(CFG_EINVAL, "amg: the hierarchy is not set up (amgValues)");
    AmgState& a = *amg_;
    const int n = dm_.nC;
    const DMat A{n, dm_.mStart, dm_.mCol};
    const int sweeps = a.decoupled ? kSingleSweeps : 0;
    // with `form`, r and p alternate between two vectors each: the kernels
    // that form them read the old values at their neighbours
    const bool form = n <= kFormRows;
    double* const rr[2] = {cr_, br_.c[0]};
    double* const pp[2] = {cp_, br_.c[1]};
    double* z = cz_;
    double* q = cAp_;
    if (!a.st)
    {
        a.st = alloc<FcgState>(1);
        CFG_CUDA(cudaMallocHost(&a.stHost, sizeof(FcgState)));
    }
    FcgState init{};
    init.tol = tol;
    init.maxIter = maxIter;
    init.normType = normType;
    CFG_CUDA(cudaMemcpyAsync(a.st, &init, sizeof(FcgState), cudaMemcpyHostToDevice, stream_));
    auto spmvInit = [&](auto Wc) {
        constexpr int W = decltype(Wc)::value;
        k_fcgd_init<W><<<GS_, TPB, 0, stream_>>>(A, vals, b, x, rr[0], partials_, a.st);
    };
    const int Wsel = maxW_ <= 7 ? 7 : (maxW_ <= 16 ? 16 : 0);
    if (Wsel == 7) spmvInit(std::integral_constant<int, 7>{});
    else if (Wsel == 16) spmvInit(std::integral_constant<int, 16>{});
    else spmvInit(std::integral_constant<int, 0>{});
    launchCheck("fcgd_init");
    amgCycle(rr[0], z, nullptr, a.st, sweeps);
    CFG_CUDA(cudaMemsetAsync(pp[0], 0, static_cast<size_t>(n) * sizeof(double), stream_));
    const auto pick = [&](auto a7, auto a16, auto a0) { return Wsel == 7 ? a7 : (Wsel == 16 ? a16 : a0); };
    const auto spmv = form ? pick(k_fcgd_spmv<7, true>, k_fcgd_spmv<16, true>, k_fcgd_spmv<0, true>)
                           : pick(k_fcgd_spmv<7, false>, k_fcgd_spmv<16, false>, k_fcgd_spmv<0, false>);
    const auto update = pick(k_fcgd_update_pre0<7>, k_fcgd_update_pre0<16>, k_fcgd_update_pre0<0>);
    const int spmvGrid = waveGrid(reinterpret_cast<const void*>(spmv), sms_, n);
    const int updateGrid = waveGrid(reinterpret_cast<const void*>(update), sms_, n);
    // iteration k of a chunk; every chunk but a solve's last has an even
    // number of them, so each begins with the vectors of index 0
    auto iteration = [&](int k) {
        const int o = form ? k & 1 : 0, w = form ? o ^ 1 : 0;
        if (!form) launchK(amgPdl(), k_fcgd_p, GS_, TPB, 0, stream_, n, z, pp[0], a.st);
        launchK(amgPdl(), spmv, spmvGrid, TPB, 0, stream_, A, vals, z, pp[o], pp[w], rr[o], q, partials_, a.st);
        if (form)
            launchK(amgPdl(), update, updateGrid, TPB, 0, stream_, A, a.vals32, a.lv[0].dinv, pp[w], q, x, rr[o], rr[w],
                    a.lv[0].x, a.lv[0].r, partials_, a.st);
        else launchK(amgPdl(), k_fcgd_update, GS_, TPB, 0, stream_, n, pp[0], q, x, rr[0], partials_, a.st);
        amgCycle(rr[w], z, q, a.st, sweeps, form);
        launchCheck("fcgd_iter", form ? 1 : 3);
    };
    for (int launched = 0, chunk = 8;;)
    {
        CFG_CUDA(cudaMemcpyAsync(a.stHost, a.st, sizeof(FcgState), cudaMemcpyDeviceToHost, stream_));
        CFG_CUDA(cudaStreamSynchronize(stream_));
        if (a.stHost->done || launched >= maxIter) break;
        const int m = std::min(chunk, maxIter - launched);
        const std::pair<std::pair<const void*, const void*>, int> key{{vals, x}, m};
        cudaGraphExec_t ge = nullptr;
        for (auto& g : a.graphs)
            if (g.first == key) ge = g.second;
        // every chunk counts its kernels once, replayed or eager
        const int64_t counted = launches_;
        if (!ge && useGraphs_)
        {
            cudaGraph_t g = nullptr;
            CFG_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
            for (int k = 0; k < m; ++k) iteration(k);
            CFG_CUDA(cudaStreamEndCapture(stream_, &g));
            const cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
            cudaGraphDestroy(g);
            if (e != cudaSuccess) fail(CFG_ECUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
            a.graphs.push_back({key, ge});
        }
        if (ge) CFG_CUDA(cudaGraphLaunch(ge, stream_));
        else
            for (int k = 0; k < m; ++k) iteration(k);
        launches_ = counted + static_cast<int64_t>(m) * ((form ? 1 : 3) + amgCycleKernels(kAmgPressure, sweeps));
        launched += m;
        chunk = std::min(chunk * 2, 32);
    }
    rep->iterations = a.stHost->it;
    rep->converged = a.stHost->conv;
    rep->initial_residual = a.stHost->init;
    rep->final_residual = a.stHost->rn;
}

void Ctx::amgInfo(double* out)
{
    // out: levels, rows of each of up to 8 levels, setup ms, values ms
    for (int k = 0; k < 11; ++k) out[k] = 0;
    if (!amg_) return;
    out[0] = static_cast<double>(amg_->lv.size());
    for (size_t l = 0; l < amg_->lv.size() && l < 8; ++l) out[1 + l] = amg_->lv[l].n;
    out[9] = amg_->setupMs;
    out[10] = amg_->valuesMs;
}

}  // namespace cfg
