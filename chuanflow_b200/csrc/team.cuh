// Teams of thread blocks that stay resident for a whole linear solve: a
// thread-block cluster (barrier.cluster, partial sums exchanged through
// distributed shared memory) or a cooperative grid (a counter barrier in
// global memory).  A Krylov iteration inside one kernel replaces three to
// seven launches, each of which costs a launch, a drain and a last-block
// reduction; on a system of a few thousand rows those are all the time.
//
// Both teams give the same services to the solver bodies (persist.cuh):
// sync(), after which every block sees what the others wrote before it, and
// reduce(), which hands the sums and maxima of per-row values to warp 0 of
// every block, where the solver's scalars advance (redundantly in each block,
// one component per lane: an FP64 division is a chain of several hundred
// cycles, and in every thread one after another they took a quarter of an
// iteration).
//
// A sum is formed in the order of the per-iteration kernels with one row per
// thread (block_sum and final_sum of dev.cuh): a tree over each 256
// consecutive rows, then a tree over those partials.  A team's blocks hold
// whole groups of 256 rows, so a solve gives the same bits in either form.
// The scalar equations of the RANS models, which stop at a fixed 1e-8, depend
// on that: another order moves their fields by a few 1e-9.

#pragma once

#include "dev.cuh"

namespace cfg
{

constexpr int kTeamThreads = 512;  // 128 registers per thread, one block per SM
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kTeamVals = 9;     // most values one reduction carries
constexpr int kTeamSums = 6;     // most of them sums
constexpr int kClusterMax = 16;  // blocks of the largest cluster (non-portable size)
constexpr int kGroupRows = TPB;  // rows of one partial sum
constexpr int kTeamRowsMax = 4;  // rows per thread (two partials each per block)
constexpr int kPartMax = 2 * kTeamRowsMax;
constexpr int kGridFold = 4;     // partials per thread of a grid team's final sum
constexpr int kGroupsMax = 256 * kGridFold;  // most groups of a system
static_assert(kGridFold == 4 && kGridFold <= FU, "team_final adds the partials in partial_sum's pairs");

/// Magnitude as an ordered integer: larger magnitudes compare larger and a
/// NaN above every number, so one integer maximum carries both |v|inf and
/// whether a NaN was seen.
__device__ __forceinline__ unsigned long long mag_bits(double v)
{
    return static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffULL;
}
__device__ __forceinline__ double mag_value(unsigned long long b)
{
    return __longlong_as_double(static_cast<long long>(b));
}

/// The teams of a launch (one per component of a solve whose components
/// iterate on their own) and the global-memory side of grid teams: per team
/// an arrival counter, an exit counter that resets them for the next launch,
/// the words of a start that no cooperative launch vouches for, and two sets of
/// partials; a flag for a wait that ran out (kTeam...), and the GPU cycles after
/// which it does.
constexpr int kTeamsMax = 3;
constexpr int kCountStride = 64;  // a team's counters on lines of their own
struct TeamMem
{
    int blocks;        // per team
    unsigned* count;   // [team][kCountStride]: arrivals at 0, exits at 32, a start's arrivals and verdict at 33, 34
    double* part;      // [team][2][kTeamVals][groups]
    int groups;        // 256-row groups of the system
    int perBlock;      // and of one block
    int* failed;
    long long wait;
    long long start;   // 0: a cooperative launch; else a plain one, whose blocks wait this long for all to be there
};
constexpr int kTeamWaitRanOut = 1, kTeamNotStarted = 2;

struct TeamSmem
{
    double warp[16][kTeamWarps];
    double mine[2][kTeamSums][kPartMax];  // this block's partial sums (read by the cluster's other blocks)
    double top[3][kTeamVals];             // and maxima; the team's
    double tree[kTeamSums][8];
    int dead;
};

template <int W>
__device__ __forceinline__ double xor_sum(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int W>
__device__ __forceinline__ double xor_max(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1)
    {
        const double w = __shfl_xor_sync(0xffffffffu, v, o);
        if (mag_bits(w) > mag_bits(v)) v = w;
    }
    return v;
}

/// Warp sums (those below NS) and maxima of P values, P a power of two, by
/// halving: at each step a lane keeps half of the values it holds and passes
/// the other half to its partner, so eight values take 9 shuffles, not 40 (in
/// a block of 16 warps the shuffles of six values one by one filled a
/// thousand cycles).  On return v[0] is value `index`.
template <int P, int NS, int O>
__device__ __forceinline__ void warp_halve(double (&v)[P], int& index)
{
    const bool up = threadIdx.x & O;
    if constexpr (P == 1)
    {
        const double w = __shfl_xor_sync(0xffffffffu, v[0], O);
        if (index < NS) v[0] += w;
        else if (mag_bits(w) > mag_bits(v[0])) v[0] = w;
        if constexpr (O > 1) warp_halve<1, NS, O / 2>(v, index);
    }
    else
    {
        double keep[P / 2];
#pragma unroll
        for (int k = 0; k < P / 2; ++k)
        {
            const double w = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[P / 2 + k], O);
            const double own = up ? v[P / 2 + k] : v[k];
            const bool sum = index + (up ? P / 2 : 0) + k < NS;
            keep[k] = sum ? own + w : (mag_bits(w) > mag_bits(own) ? w : own);
        }
        if (up) index += P / 2;
        if constexpr (O > 1) warp_halve<P / 2, NS, O / 2>(keep, index);
        v[0] = keep[0];
    }
}

/// The block's part of a reduction of K rows per thread: in warp 0, the sums
/// of 256-row group 2 k + h to sm.mine[par][q][2 k + h] and the maxima to
/// sm.top[par].
template <int K, int NS, int NM>
__device__ __forceinline__ void team_block_reduce(TeamSmem& sm, int par, const double (&s)[K][NS],
                                                  const unsigned long long (&m)[NM])
{
    constexpr int S = K * NS, N = S + NM, P = N <= 1 ? 1 : (N <= 2 ? 2 : (N <= 4 ? 4 : (N <= 8 ? 8 : 16)));
    static_assert(N <= 16 && NS <= kTeamSums && NS + NM <= kTeamVals, "team reduction too wide");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        double w[P];
#pragma unroll
        for (int i = 0; i < P; ++i)
            w[i] = i < S ? s[i < S ? i / NS : 0][i < S ? i % NS : 0] : (i < N ? mag_value(m[i < N && i >= S ? i - S : 0]) : 0.0);
        int index = 0;
        warp_halve<P, S, 16>(w, index);
        if (index < N) sm.warp[index][warp] = w[0];  // the lanes that hold a value hold the same one
    }
    __syncthreads();
    if (warp != 0) return;
    // block_sum's tree over the 8 warps of a group: lanes 0-7 and 8-15 of a
    // half warp hold the two groups of one (row slot, value)
#pragma unroll
    for (int i = 0; i < S; i += 2)
    {
        const int j = i + (lane >> 4);
        double u = j < S ? sm.warp[j][lane & 15] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
        if ((lane & 7) == 0 && j < S) sm.mine[par][j % NS][2 * (j / NS) + ((lane >> 3) & 1)] = u;
    }
#pragma unroll
    for (int q = 0; q < NM; ++q)
    {
        const double u = xor_max<kTeamWarps>(sm.warp[S + q][lane & (kTeamWarps - 1)]);
        if (lane == 0) sm.top[par][q] = u;
    }
    __syncwarp();
}

/// final_sum over the partials, from the barrier that made them visible on:
/// its thread t holds partials t, t + 256, ...; a tree over the lanes of
/// each of its eight warps here, one over the eight in warp 0, which calls f.
/// sum(q, b) is partial b of sum q, top(q, b) block b's maximum q; all of a
/// warp's loads are under way before the first is used.
template <int kFold, int NS, int NM, class Sum, class Top, class F>
__device__ __forceinline__ void team_final(TeamSmem& sm, int groups, int nb, Sum sum, Top top, F&& f)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 8)
    {
        if (32 * warp < groups)
        {
            const int t = threadIdx.x;
            double a[NS][kFold];
#pragma unroll
            for (int q = 0; q < NS; ++q)
#pragma unroll
                for (int k = 0; k < kFold; ++k) a[q][k] = sum(q, min(t + 256 * k, groups - 1));
#pragma unroll
            for (int q = 0; q < NS; ++q)
            {
#pragma unroll
                for (int k = 0; k < kFold; ++k) a[q][k] = t + 256 * k < groups ? a[q][k] : 0.0;
                // partial_sum's pairs
                double w = a[q][0];
                if constexpr (kFold == 4) w = (a[q][0] + a[q][1]) + (a[q][2] + a[q][3]);
                w = xor_sum<32>(w);
                if (lane == 0) sm.tree[q][warp] = w;
            }
        }
        else if (lane < NS) sm.tree[lane][warp] = 0.0;
    }
    else if (warp == 8 && NM > 0)
    {
#pragma unroll
        for (int q = 0; q < NM; ++q)
        {
            double v = 0.0;
            for (int k = lane; k < nb; k += 32)
            {
                const double w = top(q, k);
                if (mag_bits(w) > mag_bits(v)) v = w;
            }
            v = xor_max<32>(v);
            if (lane == 0) sm.top[2][q] = v;
        }
    }
    __syncthreads();
    if (warp == 0)
    {
        double v[NS + NM];
#pragma unroll
        for (int q = 0; q < NS; ++q)
        {
            const double* w = sm.tree[q];
            v[q] = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
        }
#pragma unroll
        for (int q = 0; q < NM; ++q) v[NS + q] = sm.top[2][q];
        f(v);
    }
    __syncthreads();
}

/// A cluster of up to kClusterMax blocks.
struct ClusterTeam
{
    static constexpr bool kCluster = true;
    TeamSmem& sm;
    int nb, team, rank, groups, per, par = 0;
    __device__ ClusterTeam(TeamSmem& s, const TeamMem& g)
        : sm(s), nb(g.blocks), team(blockIdx.x / g.blocks), rank(blockIdx.x % g.blocks), groups(g.groups), per(g.perBlock)
    {
        sync();  // every block runs before any touches another's shared memory
    }
    __device__ __forceinline__ bool dead() const { return false; }
    __device__ __forceinline__ void sync()
    {
        if (nb == 1)
        {
            __syncthreads();
            return;
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    /// f(v) in warp 0 with the team's NS sums and NM maxima in every lane,
    /// then a block barrier
    template <int K, int NS, int NM, class F>
    __device__ __forceinline__ void reduce(const double (&s)[K][NS], const unsigned long long (&m)[NM], F&& f)
    {
        team_block_reduce<K, NS, NM>(sm, par, s, m);
        sync();
        team_final<1, NS, NM>(
            sm, groups, nb, [&](int q, int b) { return fetch(&sm.mine[par][q][b % per], b / per); },
            [&](int q, int b) { return fetch(&sm.top[par][q], b); }, f);
        par ^= 1;
    }
    /// a value of another block's shared memory (or this block's own)
    __device__ __forceinline__ double fetch(const double* p, int block) const
    {
        if (nb == 1) return *p;
        unsigned remote;
        double v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(remote)
                     : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(block));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote));
        return v;
    }
    /// No block leaves while another may still read its shared memory.
    __device__ __forceinline__ void finish() { sync(); }
};

/// A cooperative grid, one block per SM at most.  A wait that has not been
/// met after `wait` cycles marks the block dead and returns; every body checks
/// dead() after each sync and reduction, leaves without storing its solution
/// and still counts itself out, so the counters are ready for the next launch.
/// A plain launch (`start`) first sees whether every block is there: the last to
/// arrive says go, a block that has waited too long says no, the first word
/// counts, and after a no every block leaves before it has written anything.
constexpr long long kTeamWaitCycles = 4000000000LL;  // about two seconds
constexpr long long kTeamStartCycles = 2000000LL;    // about a millisecond

/// whether `seen` arrivals have reached `target`, both counted modulo 2^32
__host__ __device__ constexpr bool arrived(unsigned seen, unsigned target) { return static_cast<int>(seen - target) >= 0; }
static_assert(arrived(5u, 5u) && !arrived(4u, 5u) && arrived(3u, 0xfffffff0u) && !arrived(0xfffffff0u, 3u),
              "a count that wraps does not pass its barrier early");

struct GridTeam
{
    static constexpr bool kCluster = false;
    TeamSmem& sm;
    int nb, team, rank, groups, per, par = 0;
    unsigned* count;
    double* part0;
    int* failed;
    long long wait;
    unsigned target = 0;
    __device__ GridTeam(TeamSmem& s, const TeamMem& g)
        : sm(s), nb(g.blocks), team(blockIdx.x / g.blocks), rank(blockIdx.x % g.blocks), groups(g.groups), per(g.perBlock),
          count(g.count + team * kCountStride), part0(g.part + static_cast<size_t>(team) * 2 * kTeamVals * g.groups),
          failed(g.failed), wait(g.wait)
    {
        if (threadIdx.x == 0)
        {
            sm.dead = 0;
            if (g.start > 0 && !assembled(g.start))
            {
                sm.dead = 1;
                *static_cast<volatile int*>(failed) = kTeamNotStarted;
            }
        }
        __syncthreads();
    }
    /// one thread: whether every block of the team is running at once
    __device__ __forceinline__ bool assembled(long long limit)
    {
        unsigned* const verdict = count + kCountStride / 2 + 2;  // 0: open, 1: go, 2: no
        if (atomicAdd(count + kCountStride / 2 + 1, 1u) == static_cast<unsigned>(nb) - 1u)
            return atomicCAS(verdict, 0u, 1u) == 0u;
        const long long t0 = clock64();
        for (;;)
        {
            unsigned seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(verdict) : "memory");
            if (seen == 0u && clock64() - t0 > limit)
            {
                seen = atomicCAS(verdict, 0u, 2u);
                if (seen == 0u) return false;
            }
            if (seen != 0u) return seen == 1u;
        }
    }
    __device__ __forceinline__ bool dead() const { return sm.dead != 0; }
    /// one thread: arrive (after its own writes) and wait for the others; the
    /// arrivals are compared by their distance, which a wrapped count keeps
    __device__ __forceinline__ void arrive_wait()
    {
        if (sm.dead) return;
        __threadfence();
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        const long long t0 = clock64();
        unsigned seen;
        for (;;)
        {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if (arrived(seen, target)) break;
            if (clock64() - t0 > wait)
            {
                sm.dead = 1;
                *static_cast<volatile int*>(failed) = kTeamWaitRanOut;
                break;
            }
        }
    }
    __device__ __forceinline__ void sync()
    {
        target += static_cast<unsigned>(nb);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            arrive_wait();
        }
        __syncthreads();
    }
    template <int K, int NS, int NM, class F>
    __device__ __forceinline__ void reduce(const double (&s)[K][NS], const unsigned long long (&m)[NM], F&& f)
    {
        target += static_cast<unsigned>(nb);
        const int lane = threadIdx.x & 31;
        team_block_reduce<K, NS, NM>(sm, par, s, m);
        if (threadIdx.x < 32)
        {
            double* part = part0 + static_cast<size_t>(par) * kTeamVals * groups;
            const int b = rank * per + lane;
#pragma unroll
            for (int q = 0; q < NS; ++q)
                if (lane < per && b < groups) part[q * groups + b] = sm.mine[par][q][lane];
            if (lane < NM && rank < groups) part[(NS + lane) * groups + rank] = sm.top[par][lane];
            __syncwarp();
            if (lane == 0) arrive_wait();
        }
        __syncthreads();
        const double* part = part0 + static_cast<size_t>(par) * kTeamVals * groups;
        team_final<kGridFold, NS, NM>(
            sm, groups, min(nb, groups), [&](int q, int b) { return __ldcg(part + q * groups + b); },
            [&](int q, int b) { return __ldcg(part + (NS + q) * groups + b); }, f);
        par ^= 1;
    }
    /// The last block to leave clears the counters for the next launch.
    __device__ __forceinline__ void finish()
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            __threadfence();
            if (atomicAdd(count + kCountStride / 2, 1u) == static_cast<unsigned>(nb) - 1u)
            {
                count[0] = 0;
                for (int i = 0; i < 3; ++i) count[kCountStride / 2 + i] = 0;
                __threadfence();
            }
        }
    }
};

}  // namespace cfg
