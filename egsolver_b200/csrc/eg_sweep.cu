/*
 * eg_sweep.cu -- the sweep solver: value iteration by sweeps over the input
 * CSR, cut short by certificates of unbounded credit.
 *
 * The reference's iteration (reference src/dev_EG_alg.cu:307-381) raises the
 * credits of a vertex that player 1 wins step by step until they pass MG,
 * the sum of the worst weights of all vertices.  The finite credits are
 * final long before that: of a game with 2^17 edges they settle in some
 * tens of sweeps, while the climb to MG takes thousands to millions.  This
 * solver proves "TOP" instead of climbing to it.
 *
 * Certificate.  Let S be a set of vertices and D a number for each, such
 * that with N >= 1, for every u in S,
 *   player 0: every edge (u, v, w) has v at TOP, or v in S and
 *             D(u) >= D(v) + N w + 1;
 *   player 1: some edge (u, v, w) has that property.
 * If player 1 plays such an edge wherever it can, a play from S reaches a
 * vertex at TOP or stays in S, and then the sum of N w + 1 over any cycle is
 * at most 0 (the D cancel), so every cycle has a negative weight sum: no
 * credit suffices, and the least fixed point is TOP on S.  (The fixed point
 * is the least credit of the energy game: MG bounds every finite one.)  No
 * property of D is used, so it may come from any computation.
 *
 * D is computed by value iteration too: the condition is that of the energy
 * game with the players' parts exchanged and weights -(N w + 1).  Its values
 * settle on player 1's winning vertices as fast as the credits do on player
 * 0's.  With N > n a cycle of negative sum always gives a cycle of positive
 * dual sum, so the certificate is complete; N is 2^nshift <= 2^20, and a
 * game that is not decided by it is decided by the climb.
 *
 * Schedule (advanced by every CTA in the same way after each round):
 *   primal   sweeps of credit lifts; a round without a raise ends the solve;
 *   dual     sweeps that raise D, without a barrier between them, then a
 *            copy K = D;
 *   kill     sweeps that set K(u) = out where u's condition fails on K, until
 *            a round removes nothing: what is left is the largest S.  Its
 *            credits become TOP.  An attempt that takes too many is dropped
 *            (see advance);
 *   primal   again, longer, and so on with longer dual phases.
 * A lift of every credit reads values that are initial, raised or certified,
 * all at most the least fixed point, and a primal round without a raise and
 * without a newly certified vertex has lifted every vertex against the final
 * credits: the result is the least fixed point, as of any fair schedule.
 *
 * Layout.  The grid kernel runs one CTA per SM.  A CTA owns a contiguous part
 * of player 0's vertices and one of player 1's, cut so that 8 B per edge + 28 B
 * per vertex is the same for all (both, because whole parts of one player's
 * vertices are done early), and keeps their credits and potentials and their
 * edges in shared memory for the whole solve: a sweep reads only the
 * successors' values from L2.  Vertices of at most kLightDeg out-edges are
 * sorted by (owner, out-degree) and cut into slices of 32, a warp's lanes; a
 * slice's edges lie column by column, so a thread walks its vertex without
 * bank conflicts, shuffles or much divergence; where a CTA has few, 2, 4 or 8
 * lanes share each.  A warp's lanes share a vertex of more edges; one of more
 * than kHubEdges is cut into segments dealt to the CTA's warps.  The values that gathers read are numbered the same way (the
 * CTA's base + slot), so a slice's raises are written as whole sectors.  No
 * transpose is needed.  A game that fits one CTA runs in one, every value in
 * shared memory and __syncthreads for a barrier.
 *
 * What bounds it: instructions of the control between rounds and shared-memory
 * latency in one CTA; the chain of a sweep (edge, L2 gather, store) and the
 * barrier on games of some thousand vertices; the sectors that L2 delivers to
 * random gathers on larger ones.
 * Measured, device time of a whole solve: by frontier and dense rounds that
 * climb to MG / by a first form of this kernel (lanes sharing a vertex in
 * input order, 64-bit values, a barrier with a last arriver) / this one:
 * uniform game of 131,072 vertices 684 ms / 0.41 / 0.25 ms, of 16,381 at a
 * threshold 85 ms / 0.16 / 0.09 ms; power-law game of 2^20 vertices and 8.3 M
 * edges 9.3 s / 15.9 / 4.0 ms, of 6,007 59 ms / 1.25 / 0.25 ms; complete digraph
 * of 2,000 14.2 ms / 0.47 / 0.10 ms; 4-regular game of 1,000 4.1 ms / 0.11 /
 * 0.05 ms (one CTA).
 *
 * Credits are CT integers with TOP = Lim::top while the solve runs: OMINUS(a,
 * w) is g(a - w) with g(x) = x > MG ? TOP : max(x, 0).  With MG + max |w| <
 * TOP a TOP successor always gives TOP; g is monotone and is applied once,
 * after the min or max.  CT is int32 (TOP = 2^30) where that bound and the
 * potentials' allow, else int64 (TOP = 2^62, always enough: MG <= n 2^31).
 */
#include "eg_sweep.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

namespace eg {

constexpr int kBlock = 512;      /* threads of a CTA: registers for eight gathers in flight each */
constexpr int kWarps = kBlock / 32;
constexpr int kLightDeg = 16;    /* out-edges up to which a thread may walk a vertex */
constexpr int kHubEdges = 256;   /* out-edges above which a vertex is cut; the longest segment of most */
constexpr int kMaxTasks = 1040;  /* segments of a CTA's cut vertices           */
constexpr int kBins = 2 * (kLightDeg + 1);
constexpr int kVertexBytes = 28; /* credit, potential, its copy (8 B each), id */
/* What a CTA's tables may take beyond 8 B per edge (8.5 B with the heavy
 * vertices' heads) and 28 B per vertex: the slices' pads, at most 2 x 32 x
 * kLightDeg edges per owner, and up to 62 slots without a vertex. */
constexpr int kPadEdges = 4 * 32 * kLightDeg + 64, kPadSlots = 64, kSlackBytes = 8 * kPadEdges + 8192;
/* Sweeps of the phases; the next dual and primal phases are twice as long.
 * Measured, means over 70 games of 64 to 131,072 vertices: first dual phase 6
 * 75 us, 8 81 us; 4 74 us, but 3-5% slower on 4-regular games and on one of
 * 16,381 vertices at a threshold.  Second primal phase 32 against 16, with
 * which many games need a second attempt: 2^20 vertices 4.3 against 5.6 ms. */
constexpr int kFirstPrimal = 2, kFirstDual = 6, kSecondPrimal = 32, kMaxDual = 32, kMaxPrimal = 1 << 16;
/* Rounds that a kill phase may take in any case: 329 random games, threshold
 * games and fixtures of 64 to 2^20 vertices took 43 at most. */
constexpr int kKillRounds = 128;

/* flags of a round barrier's word */
constexpr unsigned long long kTimeoutBit = 1ull << 40, kCancelBit = 1ull << 41, kRaiseMask = kTimeoutBit - 1;

template <typename CT> struct Lim;
template <> struct Lim<int> {
    static constexpr int top = 1 << 30;      /* credit TOP; potential "out of S" */
    static constexpr int low = -(1 << 30);   /* potential of a vertex at TOP     */
    static constexpr int dual_max = 1 << 29;
    static constexpr int weight_max = 1 << 20; /* of 2^nshift |w|                */
    static constexpr int none = INT32_MAX;   /* the min over no edge             */
};
template <> struct Lim<long long> {
    static constexpr long long top = 1LL << 62;
    static constexpr long long low = -(1LL << 62);
    static constexpr long long dual_max = 1LL << 61;
    static constexpr long long weight_max = 1LL << 52;
    static constexpr long long none = INT64_MAX;
};

/* Where a solve keeps what: KIND_CTA, one CTA with every value in shared
 * memory; KIND_STAGED, the grid with each CTA's values and sliced edges in
 * shared memory; KIND_GLOBAL, the grid with one or both in global memory. */
enum { KIND_CTA, KIND_STAGED, KIND_GLOBAL };

/* A CTA's vertices: slots 0 .. V ns - 1, V = 32 >> lg, hold the light ones
 * (slice s = slots V s .., 1 << lg lanes a vertex), slots V ns + h the heavy
 * ones. */
struct Range {
    int ns, s0;              /* slices; first slice of player 1              */
    int lg, light_slots;     /* log2 of a light vertex's lanes; V ns         */
    int nh, nmed;            /* heavy vertices; those not cut (the first)    */
    int base;                /* the grid's number of slot 0                  */
    int own_smem;            /* own values, ids and offsets: shared memory   */
    int stride;              /* bytes from credits to potentials to their copy there */
    int at_vid, at_soff, at_E; /* offsets in shared memory of:               */
    const int *vid;          /* vertex of each slot, -1: none                */
    const int *soff;         /* slices' first column << 5 | columns          */
    const int2 *E;           /* sliced edges: {successor's number, weight}   */
    const int2 *head;        /* heavy vertices: {first edge in H, edges | owner << 31} */
    const int2 *H, *H2;      /* their edges: those that end by h_smem, the others */
    int h_smem;
    void *g[3];              /* grid: F, D, K by number                      */
    const long long *rp;     /* the input's row offsets                      */
    int out_bits;
    long long mg, scale;
};

/* Vertices cut into segments (in shared memory). */
struct Hubs {
    int tasks, seg;
    int first[kMaxTasks / 2];
    unsigned task[kMaxTasks]; /* hub | segment << 16                          */
    long long part[kMaxTasks];
};

/* A thread's counts.  Lifts and scanned edges are counted once per vertex,
 * when it reaches TOP or at the end: until then every primal sweep lifts it. */
struct Count {
    unsigned raised;
    unsigned sweeps, heavy_sweeps; /* primal sweeps begun, of light and of heavy vertices */
    unsigned long long changes, lifts, edges;
    __device__ __forceinline__ void settle(const long long *rp, int v, bool heavy)
    {
        const unsigned n = heavy ? heavy_sweeps : sweeps;
        lifts += n;
        edges += (unsigned long long)n * (unsigned long long)(rp[v + 1] - rp[v]);
    }
};

extern __shared__ __align__(16) unsigned char smem[];

/* One kind of sweep: which array it lifts (0: credits, 1: potentials, 2:
 * their copy) and how.  Primal: x = the min (player 0) or max (player 1) of
 * f(v) - w; dual and kill: the max or min of D(v) + scale w + 1.  All are
 * taken as a min, of `sign` x the edge's value, with sign = -1 for a max:
 *   sign y + sign mul w,  mul = -1 (primal) or scale,
 * and the result is sign x min + add. */
template <typename CT>
struct Kind {
    int mode;
    int mul;
    CT cap, add;             /* largest value short of TOP; 0 or 1           */
};

__device__ __forceinline__ int edge_value(int sign, int y, int mul, int w) { return sign * y + mul * w; }
__device__ __forceinline__ long long edge_value(int sign, long long y, int mul, int w)
{
    return (sign < 0 ? -y : y) + (long long)mul * (long long)w;
}

/* Access to the places of a KIND: own values by slot; successors' by slot in
 * one CTA, by number on the grid.  A slot without a vertex holds TOP,
 * potential LOW. */
template <typename CT, int KIND>
struct Mem {
    static __device__ __forceinline__ int vid(const Range &r, int slot)
    {
        return KIND == KIND_GLOBAL ? r.vid[slot] : *(const int *)(smem + r.at_vid + 4 * slot);
    }
    static __device__ __forceinline__ int soff(const Range &r, int s)
    {
        return KIND == KIND_GLOBAL ? r.soff[s] : *(const int *)(smem + r.at_soff + 4 * s);
    }
    static __device__ __forceinline__ CT own(const Range &r, int which, int slot)
    {
        if (KIND != KIND_GLOBAL || r.own_smem) return *(const CT *)(smem + which * r.stride + (int)sizeof(CT) * slot);
        return ((const CT *)r.g[which])[r.base + slot];
    }
    static __device__ __forceinline__ void set(const Range &r, int which, int slot, CT x)
    {
        if (KIND != KIND_GLOBAL || r.own_smem) *(CT *)(smem + which * r.stride + (int)sizeof(CT) * slot) = x;
        if (KIND == KIND_CTA) return;
        if (sizeof(CT) == 4) __stcg((int *)r.g[which] + r.base + slot, (int)x);
        else __stcg((long long *)r.g[which] + r.base + slot, (long long)x);
    }
    /* a successor's value; g, at_g: the array's global and shared place */
    static __device__ __forceinline__ CT gather(const CT *g, int at_g, int at)
    {
        if (KIND == KIND_CTA) return *(const CT *)(smem + at_g + (int)sizeof(CT) * at);
        if (sizeof(CT) == 4) return (CT)__ldcg((const int *)g + at);
        return (CT)__ldcg((const long long *)g + at);
    }
};

/* The last step of a vertex, by one thread. */
template <typename CT, int KIND>
__device__ __forceinline__ void finish_vertex(const Range &r, const Kind<CT> &k, int sign, int slot, CT old, CT acc,
                                              Count &cnt)
{
    using M = Mem<CT, KIND>;
    constexpr CT top = Lim<CT>::top;
    const CT x = (sign < 0 ? -acc : acc) + k.add;
    CT nv = x > 0 ? x : (CT)0;
    if (nv > k.cap) nv = top;
    if (nv <= old) return;
    cnt.raised++;
    if (k.mode == SWEEP_KILL) nv = top;
    M::set(r, k.mode, slot, nv);
    if (k.mode == SWEEP_PRIMAL && nv == top) {
        M::set(r, 1, slot, Lim<CT>::low);
        cnt.settle(r.rp, M::vid(r, slot), slot >= r.light_slots);
    }
}

/* Up to U columns of a slice, E at a lane's first: their loads, then the
 * gathers, then the values.  PADS: an edge may be none (-1). */
template <typename CT, int KIND, int U, bool PADS>
__device__ __forceinline__ CT walk(const int2 *E, int columns, const CT *g, int at_g, int sign, int mul, CT acc)
{
    int2 q[U];
    CT y[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
        if (PADS) q[j].x = -1;
        if (j < columns) q[j] = E[32 * j];
    }
#pragma unroll
    for (int j = 0; j < U; j++)
        if (PADS ? q[j].x >= 0 : j < columns) y[j] = Mem<CT, KIND>::gather(g, at_g, q[j].x);
#pragma unroll
    for (int j = 0; j < U; j++)
        if (PADS ? q[j].x >= 0 : j < columns) acc = min(acc, edge_value(sign, y[j], mul, q[j].y));
    return acc;
}

/* Loads in flight per lane: a few for shared-memory gathers, enough to cover
 * an L2 gather for all but the longest rows. */
template <int KIND> constexpr int kUnroll = KIND == KIND_CTA ? 2 : 8;
constexpr int kGroupUnroll = 4; /* where lanes share a vertex, most walk no further */

/* The heavy vertices of one sweep: first the segments of those that are cut,
 * then a warp per vertex of the others (the warps with the fewest slices
 * first), then the cut ones' results. */
template <typename CT, int KIND>
__device__ __forceinline__ void sweep_heavy(const Range &r, const Kind<CT> &kd, Hubs &hb, Count &cnt)
{
    using M = Mem<CT, KIND>;
    constexpr int U = kUnroll<KIND>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot0 = r.light_slots;
    const bool hubs = r.nh > r.nmed;
    const CT *g = (const CT *)r.g[kd.mode];
    const int at_g = kd.mode * r.stride;
    int2 hd;
    const int2 *H;
    int sign;
    CT old;
    auto open = [&](int h) {
        old = M::own(r, kd.mode, slot0 + h);
        if (old >= Lim<CT>::top || old == Lim<CT>::low) return false;
        hd = r.head[h];
        sign = (hd.y < 0) == (kd.mode == SWEEP_PRIMAL) ? -1 : 1;
        hd.y &= INT32_MAX;
        H = (hd.x + hd.y <= r.h_smem ? r.H : r.H2) + hd.x;
        return true;
    };
    auto batch = [&](auto u, int k, int k1, CT acc) {
        /* past the end: the last edge again, which changes no min (a look at
         * each edge instead: complete digraph of 2,000 183 -> 153 us without,
         * most of it registers that were spilled) */
        constexpr int N = decltype(u)::value;
        int2 q[N];
        CT y[N];
#pragma unroll
        for (int j = 0; j < N; j++) q[j] = H[min(k + 32 * j, k1 - 1)];
#pragma unroll
        for (int j = 0; j < N; j++) y[j] = M::gather(g, at_g, q[j].x);
#pragma unroll
        for (int j = 0; j < N; j++) acc = min(acc, edge_value(sign, y[j], sign * kd.mul, q[j].y));
        return acc;
    };
    /* Short remainders in short batches, as most heavy vertices of a power-law
     * game are: 2^20 vertices 4.2-5.6 -> 3.7-4.2 ms. */
    auto lanes_min = [&](int k0, int k1) {
        CT acc = Lim<CT>::none;
#pragma unroll 1
        for (int k = k0 + lane; k - lane < k1; k += 32 * U) {
            const int left = k1 - (k - lane);
            if (left > 64) acc = batch(std::integral_constant<int, U>(), k, k1, acc);
            else if (left > 32) acc = batch(std::integral_constant<int, 2>(), k, k1, acc);
            else acc = batch(std::integral_constant<int, 1>(), k, k1, acc);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc = min(acc, (CT)__shfl_xor_sync(0xffffffffu, acc, o));
        return acc;
    };
    if (hubs) {
        for (int t = warp; t < hb.tasks; t += kWarps) {
            const unsigned tk = hb.task[t];
            if (!open(r.nmed + (int)(tk & 0xffffu))) continue;
            const int k0 = (int)(tk >> 16) * hb.seg;
            const CT acc = lanes_min(k0, min(hd.y, k0 + hb.seg));
            if (lane == 0) hb.part[t] = (long long)acc;
        }
    }
    for (int h = (warp - r.ns) & (kWarps - 1); h < r.nmed; h += kWarps) {
        if (!open(h)) continue;
        const CT acc = lanes_min(0, hd.y);
        if (lane == 0) finish_vertex<CT, KIND>(r, kd, sign, slot0 + h, old, acc, cnt);
    }
    if (hubs) {
        __syncthreads();
        for (int h = r.nmed + warp; h < r.nh; h += kWarps) {
            if (!open(h)) continue;
            const int nt = (hd.y + hb.seg - 1) / hb.seg, t0 = hb.first[h - r.nmed];
            CT acc = Lim<CT>::none;
            for (int t = lane; t < nt; t += 32) acc = min(acc, (CT)hb.part[t0 + t]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc = min(acc, (CT)__shfl_xor_sync(0xffffffffu, acc, o));
            if (lane == 0) finish_vertex<CT, KIND>(r, kd, sign, slot0 + h, old, acc, cnt);
        }
        __syncthreads();
    }
}

/* One sweep of the CTA's vertices: the light ones here, a slice per warp, a
 * vertex per lane. */
template <typename CT, int KIND, bool GROUP>
__device__ __forceinline__ void sweep(const Range &r, const Kind<CT> &kd, Hubs &hb, Count &cnt, bool heavy)
{
    using M = Mem<CT, KIND>;
    constexpr int U = kUnroll<KIND>;
    const int lane = threadIdx.x & 31;
    const CT *g = (const CT *)r.g[kd.mode];
    const int at_g = kd.mode * r.stride;
    if (const int s = threadIdx.x >> 5; GROUP && s < r.ns) { /* no more slices than warps */
        const int slot = (32 * s + lane) >> r.lg;
        const int x = M::soff(r, s);
        const int sign = (s >= r.s0) == (kd.mode == SWEEP_PRIMAL) ? -1 : 1;
        const CT old = M::own(r, kd.mode, slot);
        const bool live = old < Lim<CT>::top && old != Lim<CT>::low;
        const int2 *E = KIND == KIND_GLOBAL ? r.E + 32 * (long long)(x >> 5) + lane
                                            : (const int2 *)(smem + r.at_E) + 32 * (x >> 5) + lane;
        CT acc = Lim<CT>::none;
#pragma unroll 1
        for (int left = live ? x & 31 : 0; left > 0; left -= kGroupUnroll, E += 32 * kGroupUnroll)
            acc = walk<CT, KIND, kGroupUnroll, true>(E, left, g, at_g, sign, sign * kd.mul, acc);
        __syncwarp();
        for (int o = 1 << r.lg >> 1; o > 0; o >>= 1) acc = min(acc, (CT)__shfl_xor_sync(0xffffffffu, acc, o));
        if (live && (lane & ((1 << r.lg) - 1)) == 0) finish_vertex<CT, KIND>(r, kd, sign, slot, old, acc, cnt);
        __syncwarp();
    }
    for (int s = threadIdx.x >> 5; !GROUP && s < r.ns; s += kWarps) {
        const int slot = 32 * s + lane;
        const int x = M::soff(r, s);
        const int sign = (s >= r.s0) == (kd.mode == SWEEP_PRIMAL) ? -1 : 1;
        const CT old = M::own(r, kd.mode, slot);
        if (old >= Lim<CT>::top || old == Lim<CT>::low) continue;
        const int2 *E = KIND == KIND_GLOBAL ? r.E + 32 * (long long)(x >> 5) + lane
                                            : (const int2 *)(smem + r.at_E) + 32 * (x >> 5) + lane;
        CT acc = Lim<CT>::none;
#pragma unroll 1
        /* full batches apart: 131,072 vertices 262 -> 248 us */
        for (int left = x & 31; left > 0; left -= U, E += 32 * U) {
            if (left >= U) acc = walk<CT, KIND, U, false>(E, U, g, at_g, sign, sign * kd.mul, acc);
            else acc = walk<CT, KIND, U, false>(E, left, g, at_g, sign, sign * kd.mul, acc);
        }
        finish_vertex<CT, KIND>(r, kd, sign, slot, old, acc, cnt);
    }
    if (heavy && r.nh) sweep_heavy<CT, KIND>(r, kd, hb, cnt);
}

/* The schedule after a round of `ran` sweeps in which `raised` values changed
 * (any number but 0 where it is only compared with that).  `stop`: the time
 * limit or the cancel flag, which ends any phase: the credits are lower bounds
 * at all times.  Returns whether what is left of S is certified.
 *
 * A kill phase may be as long as the game is deep, and on a path certifies
 * nothing: it is dropped once it has cost as much as the credits so far, and
 * what follows an attempt is at least as long as it was, so that kills stay
 * within about one and a half times the primal rounds (path of 16,384 vertices
 * 52 ms; kills to their end 239 ms, ten times the primal sweeps). */
__device__ __forceinline__ bool advance(const SweepParams &p, SweepState &c, int ran, unsigned long long raised, int stop)
{
    if (c.phase == SWEEP_PRIMAL) {
        c.rounds++;
        c.sweeps += ran;
        c.left -= ran;
        if (raised == 0ull) {
            c.phase = SWEEP_DONE;
            return false;
        }
        if (p.max_rounds >= 0 && c.rounds >= p.max_rounds) stop = (int)EG_ERR_LOOPCAP;
        c.stop = stop;
        if (stop || c.left > 0) return false;
        if (p.hand_sweeps && c.sweeps >= p.hand_sweeps && (long long)raised < p.hand_raised) {
            c.phase = SWEEP_HANDOVER;
            return false;
        }
        c.phase = SWEEP_DUAL;
        c.left = c.dual_len;
        return false;
    }
    c.stop = stop;
    /* rounds of a kill phase: `left` counts them down (`rounds` stands still) */
    const int most = (int)max((long long)kKillRounds, min(c.rounds, 1ll << 28));
    if (c.phase == SWEEP_DUAL) {
        c.dual_len = min(2 * c.dual_len, kMaxDual);
        c.phase = SWEEP_KILL;
        c.left = most;
        return false;
    }
    if (raised != 0ull && --c.left > 0) return false;
    const bool certified = raised == 0ull;
    const int kills = most - c.left;
    c.phase = SWEEP_PRIMAL;
    c.left = c.primal_len;
    if (kills >= kKillRounds) c.left = max(c.left, (certified ? 2 : 4) * kills);
    c.primal_len = min(2 * c.primal_len, kMaxPrimal);
    return certified;
}

__device__ __forceinline__ unsigned long long ld_acquire_gpu64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* Round barrier `it` of the grid (thread 0 of each CTA): one atomic carries
 * the arrival, this CTA's raises and (CTA 0) the stop flags, and everybody
 * polls that word until all have arrived, so it also brings the sum of the
 * raises: one round trip and a poll, 2,400 cycles with 148 CTAs (a flag per
 * CTA that all poll: 4,500 to 7,300; a last arriver that publishes a decision:
 * about 10,000).  Words are used in turn; word it + 2 was last read at
 * barrier it - 2, which all CTAs have left.  Bounded by wait_limit_ns; returns
 * false when a CTA gave up. */
__device__ __forceinline__ bool round_barrier(const SweepParams &p, SweepCtrl *c, unsigned it, unsigned long long give,
                                              unsigned long long *sum)
{
    unsigned long long *w = &c->word[it & 3][0];
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"((1ull << 48) | give) : "memory");
    unsigned long long v, t0 = 0;
    unsigned spins = 0;
    while (((v = ld_acquire_gpu64(w)) >> 48) != gridDim.x) {
        if ((++spins & 255) == 0) {
            if (ld_volatile(&c->abort)) return false;
            const unsigned long long now = globaltimer_ns();
            if (!t0) t0 = now;
            else if (now - t0 > p.wait_limit_ns) {
                c->wait_site = it;
                atomicExch(&c->abort, 1);
                return false;
            }
        }
    }
    if (blockIdx.x == 0) c->word[(it + 2) & 3][0] = 0ull;
    *sum = v & ((1ull << 48) - 1);
    return true;
}

/* What a CTA's threads tell each other at the end of a round. */
struct Turn {
    unsigned raised[2];       /* by parity                                   */
    unsigned long long sum;   /* grid: the barrier's sum and flags           */
    int ok, stop;
};

/* Everything after the set-up, for one credit width and kind.  Not inlined:
 * each has its registers to itself. */
template <typename CT, int KIND, bool GROUP>
__device__ __noinline__ void solve(const SweepParams *pp, const Range &rs, Hubs &hb, Turn &turn, SweepState &state,
                                   unsigned it, Count &count)
{
    using M = Mem<CT, KIND>;
    constexpr bool GRID = KIND != KIND_CTA;
    /* primal and kill sweeps between two barriers (with four, more of them come
     * after the last raise) */
    constexpr int kRound = GRID ? 2 : 1;
    constexpr CT top = Lim<CT>::top, low = Lim<CT>::low;
    const SweepParams &p = *pp;
    /* in registers where lanes walk long slices; the code without those is
     * faster with them in shared memory (complete digraph 171 -> 152 us) */
    std::conditional_t<GROUP, const Range &, const Range> r = rs;
    SweepState st = state;
    const unsigned first = it;
    Count cnt = count;
    const int tid = threadIdx.x, lane = tid & 31;
    const int nslots = r.light_slots + r.nh;
    const bool watch = p.timeout_ns || p.cancel;
    const bool watcher = watch && tid == 0 && blockIdx.x == 0;
    bool ok = turn.ok != 0, mark = false;
    /* slots without a vertex are never lifted (the others start at 0) */
    for (int i = tid; i < r.light_slots; i += kBlock) {
        if (M::vid(r, i) < 0) {
            M::set(r, 0, i, top);
            M::set(r, 1, i, low);
        }
    }
    __syncthreads();
    while (ok && !st.stop && st.phase < SWEEP_DONE) {
        const int phase = st.phase;
        cnt.raised = 0u;
        if (mark) { /* the certified vertices: TOP */
            for (int i = tid; i < nslots; i += kBlock) {
                const CT k = M::own(r, 2, i);
                if (k < top && k != low) {
                    M::set(r, 0, i, top);
                    M::set(r, 1, i, low);
                    cnt.raised++;
                    cnt.settle(r.rp, M::vid(r, i), i >= r.light_slots);
                }
            }
            __syncthreads();
        }
        Kind<CT> kd;
        kd.mode = phase;
        kd.mul = phase == SWEEP_PRIMAL ? -1 : (int)r.scale;
        kd.cap = phase == SWEEP_PRIMAL ? (CT)r.mg : Lim<CT>::dual_max;
        kd.add = phase == SWEEP_PRIMAL ? (CT)0 : (CT)1;
        const int ran = phase == SWEEP_DUAL ? st.left : phase == SWEEP_KILL || !GRID ? kRound : min(kRound, st.left);
#pragma unroll 1
        for (int s = 0; s < ran; s++) {
            /* The heavy vertices every second time, and in a round's last sweep,
             * so that a round without a raise has lifted all.  They are most of
             * the edges of a power-law game, and the parts that hold them the
             * last at every barrier, but move no faster than what they gather
             * (power-law games of 2^20 vertices 3.5-5.9 -> 2.5-4.0 ms, of up to
             * 6,000 211 -> 188 us, complete digraphs 114 -> 77).  In one CTA, with
             * no barrier to be late at, all every time. */
            const bool heavy = !GRID || s == ran - 1 || (phase == SWEEP_DUAL && (s & 1));
            if (phase == SWEEP_PRIMAL) {
                cnt.sweeps++;
                cnt.heavy_sweeps += heavy;
            }
            sweep<CT, KIND, GROUP>(r, kd, hb, cnt, heavy);
        }
        if (phase == SWEEP_PRIMAL) cnt.changes += cnt.raised;
        if (phase == SWEEP_DUAL) {
            __syncthreads();
            for (int i = tid; i < nslots; i += kBlock) M::set(r, 2, i, M::own(r, 1, i));
        }
        /* the round's raises and the next step of the schedule */
        unsigned long long raised;
        int stop = 0;
        if (watcher) {
            if (p.timeout_ns && globaltimer_ns() - p.ctrl->t_start > p.timeout_ns) stop = (int)EG_ERR_TIMEOUT;
            else if (p.cancel && ((it - first) & 63) == 0 && ld_volatile(p.cancel)) stop = (int)EG_ERR_CANCELLED;
        }
        if (GRID) {
            const unsigned d = __reduce_add_sync(0xffffffffu, cnt.raised);
            if (lane == 0 && d) atomicAdd(&turn.raised[it & 1], d);
            __syncthreads();
            if (tid == 0) {
                unsigned long long give = turn.raised[it & 1], got = 0ull;
                turn.raised[it & 1] = 0u; /* next used two rounds on */
                if (stop) give |= stop == (int)EG_ERR_TIMEOUT ? kTimeoutBit : kCancelBit;
                turn.ok = round_barrier(p, p.ctrl, it, give, &got);
                turn.sum = got;
            }
            __syncthreads();
            ok = turn.ok != 0;
            raised = turn.sum & kRaiseMask;
            stop = turn.sum & kTimeoutBit ? (int)EG_ERR_TIMEOUT : turn.sum & kCancelBit ? (int)EG_ERR_CANCELLED : 0;
        } else {
            if (tid == 0 && watch) turn.stop = stop;
            raised = (unsigned long long)__syncthreads_or((int)cnt.raised);
            if (watch) {
                stop = turn.stop;
                __syncthreads();
            }
        }
        mark = advance(p, st, ran, raised, stop);
        it++;
    }
    __syncthreads();
    /* credits out; TOPs are counted in `raised` */
    cnt.raised = 0u;
    for (int i = tid; i < nslots; i += kBlock) {
        const int v = M::vid(r, i);
        if (v < 0) continue;
        const CT f = M::own(r, 0, i);
        if (f == top) cnt.raised++;
        else cnt.settle(r.rp, v, i >= r.light_slots);
        if (r.out_bits == 32) ((int *)p.out)[v] = f == top ? INT32_MAX : (int)f;
        else ((long long *)p.out)[v] = f == top ? (long long)INT64_MAX : (long long)f;
    }
    count = cnt;
    state = st;
}

__device__ __forceinline__ unsigned long long cost_before(const SweepParams &p, long long v)
{
    return (unsigned long long)p.rp[v] * 8ull + (unsigned long long)v * kVertexBytes;
}

/* Cuts both players' vertices into gridDim.x parts of equal cost: cut[0] ..
 * cut[1] of player 0's [0, split) and cut[2] .. cut[3] of player 1's [split,
 * n) are this CTA's.  A search in which 128 threads probe places for each cut
 * at a time. */
__device__ __forceinline__ void find_cuts(const SweepParams &p, int split, int *s_probe, int *cut)
{
    const int q = threadIdx.x >> 7, t = threadIdx.x & 127;
    const int b0 = q < 2 ? 0 : split, b1 = q < 2 ? split : p.n;
    const unsigned long long c0 = cost_before(p, b0), total = cost_before(p, b1) - c0;
    const unsigned long long part = blockIdx.x + (q & 1), parts = gridDim.x;
    const unsigned long long target = c0 + total / parts * part + total % parts * part / parts;
    int lo = b0, hi = part == parts ? b0 : b1; /* the answer is in [lo, hi] */
    if (part == parts) lo = hi = b1;
    if (threadIdx.x < 4) s_probe[threadIdx.x] = 0;
    for (;;) {
        const int step = (hi - lo + 127) >> 7;
        const long long at = (long long)lo + (long long)t * step;
        const bool below = at < hi && cost_before(p, at) < target;
        const unsigned m = __ballot_sync(0xffffffffu, below);
        if (!__syncthreads_or(lo < hi)) break;
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(&s_probe[q], __popc(m));
        __syncthreads();
        const int c = s_probe[q]; /* probes below the target: the first c */
        __syncthreads();
        if (threadIdx.x < 4) s_probe[threadIdx.x] = 0;
        if (lo < hi) {
            const long long next = (long long)lo + (long long)c * step;
            if (c > 0) lo = (int)((long long)lo + (long long)(c - 1) * step + 1);
            if (next < hi) hi = (int)next;
        }
    }
    if (t == 0) s_probe[q] = lo;
    __syncthreads();
    for (int k = 0; k < 4; k++) cut[k] = s_probe[k];
    __syncthreads();
}

template <bool GRID>
__global__ void __launch_bounds__(kBlock, 1) k_sweep(const __grid_constant__ SweepParams p)
{
    __shared__ Hubs hb;
    __shared__ Turn turn;
    __shared__ Range r;
    __shared__ SweepParams ps;
    __shared__ unsigned long long s_sum[4]; /* MG, largest |weight|; then TOPs, lifts, edges, raises */
    __shared__ int s_bin[kBins];            /* light vertices by owner and out-degree, then their next slot */
    __shared__ int s_cls[5];                /* first slot past the light vertices of player 0; of player 1; columns; light; lg */
    __shared__ int s_heavy[4];              /* heavy vertices: not cut, cut; their edges; next offset */
    __shared__ int s_scan[kWarps];
    __shared__ int s_sink;                  /* a vertex has no successor: the walks count on one */
    SweepCtrl *c = p.ctrl;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    /* with an owner array the players' vertices are not apart: one part */
    const int split = p.owner ? p.n : p.n0;
    int cut[4] = {0, split, split, p.n};
    if (GRID) find_cuts(p, split, s_heavy, cut);
    const int nv0 = cut[1] - cut[0], nv = nv0 + cut[3] - cut[2];
    const int gap = cut[2] - nv0; /* vertex i of the CTA: cut[0] + i, or gap + i from nv0 on */
    const long long e0 = p.rp[cut[0]], e1 = p.rp[cut[2]];
    const int ne = (int)(p.rp[cut[1]] - e0 + p.rp[cut[3]] - e1);
    /* Vertices of more than `cut_from` edges are cut, so that each warp has
     * one of their segments (power-law games of 6,000 vertices: 269 -> 254 us,
     * 412 -> 330 us against segments of 256), into at most 512 + 512 of them. */
    const int cut_from = max(kHubEdges, (ne / 512 + 31) & ~31);
    const int seg = ne >= 512 * kHubEdges ? cut_from : min(kHubEdges, max(64, (ne / kWarps + 31) & ~31));
    __syncthreads();
    if (tid < kBins) s_bin[tid] = 0;
    if (tid < 4) {
        s_sum[tid] = 0ull;
        s_heavy[tid] = 0;
    }
    if (tid == 0) {
        if (blockIdx.x == 0) c->t_start = globaltimer_ns();
        s_sink = 0;
        hb.tasks = 0;
        hb.seg = seg;
        turn.raised[0] = turn.raised[1] = 0u;
        turn.sum = 0ull;
        turn.ok = 1;
        turn.stop = 0;
    }
    __syncthreads();
    /* 1. vertices by kind */
    for (int i = tid; i < nv; i += kBlock) {
        const int v = i < nv0 ? cut[0] + i : gap + i;
        const int deg = (int)(p.rp[v + 1] - p.rp[v]);
        if (deg <= 0) s_sink = 1;
        if (deg <= kLightDeg) {
            const int own1 = p.owner ? p.owner[v] != 0 : v >= p.n0;
            atomicAdd(&s_bin[own1 * (kLightDeg + 1) + max(deg, 0)], 1);
        } else {
            atomicAdd(&s_heavy[deg > cut_from], 1);
            atomicAdd(&s_heavy[2], deg);
        }
    }
    __syncthreads();
    if (tid < 2) {
        /* Up to how many out-edges a thread walks a vertex: a warp's second
         * batch of loads (columns 9 to 16) costs another L2 latency, so where
         * the vertices that need it find a warp each beside the slices, they
         * get one (games of 4,000 to 6,000 vertices: 215 -> 133 us, 510 -> 425
         * us; of 16,000, whose CTAs have too many, 143 -> 239 us). */
        int few[2] = {0, 0}, many = 0, edges = 0;
        for (int o = 0; o < 2; o++) {
            for (int d = 0; d <= kLightDeg; d++) {
                const int x = s_bin[o * (kLightDeg + 1) + d];
                few[o] += d <= kLightDeg / 2 ? x : 0;
                many += d > kLightDeg / 2 ? x : 0;
                edges += d > kLightDeg / 2 ? d * x : 0;
            }
        }
        /* Lanes of a light vertex: as many as leave every slice and every
         * heavy vertex a warp of its own, and no more than it has out-edges.
         * A sweep of a few hundred edges is one warp's chain of loads and
         * instructions, which shared rows shorten (games of 2,000 vertices
         * 85 -> 60 us, 5,000 112 -> 72, 16,000 118 -> 87; in one CTA, with
         * gathers from shared memory, 2 us longer). */
        int all[2], lg = GRID ? 3 : 0, most = 0;
        for (int o = 0; o < 2; o++) {
            all[o] = 0;
            for (int d = 0; d <= kLightDeg; d++) {
                const int x = s_bin[o * (kLightDeg + 1) + d];
                all[o] += x;
                if (x) most = max(most, d);
            }
        }
        while (lg && ((1 << lg >> 1) >= most ||
                      ((all[0] + (31 >> lg)) >> (5 - lg)) + ((all[1] + (31 >> lg)) >> (5 - lg)) + s_heavy[0] > kWarps))
            lg--;
        const bool half = !lg && ((few[0] + 31) >> 5) + ((few[1] + 31) >> 5) + s_heavy[0] + many <= kWarps;
        const int light = half ? kLightDeg / 2 : kLightDeg;
        __syncwarp(3u);
        if (half && tid == 0) {
            s_heavy[0] += many;
            s_heavy[2] += edges;
        }
        if (tid == 0) {
            s_cls[3] = light;
            s_cls[4] = lg;
        }
        /* the first slot of every (owner, out-degree); player 1's start a slice */
        int total0 = 0;
        for (int d = 0; d <= light; d++) total0 += s_bin[d];
        int at = tid ? (total0 + (31 >> lg)) & ~(31 >> lg) : 0;
        __syncwarp(3u);
        for (int d = 0; d <= light; d++) {
            const int k = tid * (kLightDeg + 1) + d, x = s_bin[k];
            s_bin[k] = at;
            at += x;
        }
        s_cls[tid] = at;
    }
    __syncthreads();
    const int light = s_cls[3], lg = s_cls[4], V = 32 >> lg;
    const int nmed = s_heavy[0], nh = nmed + s_heavy[1], he = s_heavy[2];
    /* 2. shared memory: own values, ids, slice offsets; then sliced edges;
     * then heavy ones -- what does not fit is in global memory */
    const int s0 = (s_cls[0] + V - 1) >> (5 - lg), ns = (s_cls[1] + V - 1) >> (5 - lg), nslots = V * ns + nh;
    const int stride = 8 * nslots;
    const int base = GRID ? cut[0] + cut[2] - split + kPadSlots * (int)blockIdx.x : 0;
    long long at = 28LL * nslots + 4LL * ns;
    const bool own_smem = at <= p.smem_bytes;
    int *vid, *soff;
    if (own_smem) {
        vid = (int *)(smem + 3 * stride);
        soff = vid + nslots;
        at = (at + 15) & ~15LL;
    } else {
        vid = p.vid + base;
        soff = p.soff + (base >> 5) + 4 * (long long)blockIdx.x;
        at = 0;
    }
    /* slice widths: the out-degree of a slice's last vertex; their sums */
    {
        int run = 0;
        for (int first = 0; first < ns; first += kBlock) {
            const int s = first + tid;
            int W = 0;
            if (s < ns) {
                const int own1 = s >= s0;
                const int last = min(V * s + V - 1, s_cls[own1] - 1);
                for (int d = 1; d <= light; d++) W += s_bin[own1 * (kLightDeg + 1) + d] <= last;
                W = (W + (1 << lg) - 1) >> lg;
            }
            int x = W;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_scan[warp] = x;
            __syncthreads();
            int before = 0, all = 0;
            for (int k = 0; k < kWarps; k++) {
                before += k < warp ? s_scan[k] : 0;
                all += s_scan[k];
            }
            if (s < ns) soff[s] = (run + before + x - W) << 5 | W;
            run += all;
            __syncthreads();
        }
        if (tid == 0) s_cls[2] = run;
    }
    for (int i = tid; i < V * ns; i += kBlock) vid[i] = -1;
    if (own_smem)
        for (int i = tid; i < 2 * nslots; i += kBlock) ((long long *)smem)[i] = 0;
    if (GRID) {
        /* up to the next CTA's numbers: 32-bit values lie elsewhere in the arrays */
        for (int i = tid; i < nv + kPadSlots; i += kBlock) {
            __stcg((long long *)p.F + base + i, 0LL);
            __stcg((long long *)p.D + base + i, 0LL);
        }
    }
    __syncthreads();
    const long long ell = 32LL * s_cls[2]; /* edges with pads */
    const int at_E = (int)at;
    const bool edges_smem = at + 8 * ell <= p.smem_bytes;
    /* the heavy ones as far as they fit (complete digraph of 2,000, whose parts
     * are 3% too large: 217 -> 197 us against none) */
    const bool heavy_smem = at + 8 * (ell + nh) <= p.smem_bytes;
    const int h_smem = heavy_smem ? (int)min((p.smem_bytes - at) / 8 - ell - nh, (long long)he) : he;
    int2 *E, *rest = nullptr; /* where the sliced edges are, and the heavy heads and edges */
    int2 *out_of_smem = p.E + (e0 + e1 - p.rp[split]) + ((e0 + e1 - p.rp[split]) >> 4) + kPadEdges * (long long)blockIdx.x;
    E = edges_smem ? (int2 *)(smem + at) : out_of_smem;
    rest = heavy_smem ? (int2 *)(smem + at) + ell : edges_smem ? out_of_smem : out_of_smem + ell;
    int2 *head = rest, *H = rest + nh, *H2 = heavy_smem && edges_smem ? out_of_smem : H;
    if (tid < 2) s_heavy[tid] = 0;
    if (tid == 0) {
        ps = p;
        r.ns = ns;
        r.lg = lg;
        r.light_slots = V * ns;
        r.s0 = s0;
        r.nh = nh;
        r.nmed = nmed;
        r.base = base;
        r.own_smem = own_smem;
        r.stride = stride;
        r.at_vid = 3 * stride;
        r.at_soff = r.at_vid + 4 * nslots;
        r.at_E = at_E;
        r.vid = vid;
        r.soff = soff;
        r.E = E;
        r.head = head;
        r.H = H;
        r.H2 = H2;
        r.h_smem = h_smem;
        r.g[0] = p.F;
        r.g[1] = p.D;
        r.g[2] = p.K;
        r.rp = p.rp;
    }
    int *number = GRID ? (int *)p.K : (int *)(smem + 2 * stride); /* of every vertex, where K is later */
    __syncthreads();
    /* 3. slots */
    for (int i = tid; i < nv; i += kBlock) {
        const int v = i < nv0 ? cut[0] + i : gap + i;
        const int deg = (int)(p.rp[v + 1] - p.rp[v]);
        const int own1 = p.owner ? p.owner[v] != 0 : v >= p.n0;
        int slot;
        if (deg <= light) {
            slot = atomicAdd(&s_bin[own1 * (kLightDeg + 1) + max(deg, 0)], 1);
        } else {
            const int hub = deg > cut_from;
            const int h = (hub ? nmed : 0) + atomicAdd(&s_heavy[hub], 1);
            slot = V * ns + h;
            head[h] = make_int2(atomicAdd(&s_heavy[3], deg), (int)((unsigned)deg | (unsigned)own1 << 31));
            if (hub) {
                const int nt = (deg + seg - 1) / seg, t0 = atomicAdd(&hb.tasks, nt), k = h - nmed;
                hb.first[k] = t0;
                for (int t = 0; t < nt; t++) hb.task[t0 + t] = (unsigned)k | (unsigned)t << 16;
            }
        }
        vid[slot] = v;
        if (GRID) __stcg(number + v, base + slot);
        else number[v] = slot;
    }
    __syncthreads();
    unsigned it = 0;
    unsigned long long got = 0ull;
    if (GRID) { /* every vertex has its number */
        if (tid == 0) turn.ok = round_barrier(p, c, it, 0ull, &got);
        it++;
        __syncthreads();
    }
    /* 4. edges; MG and the largest |weight| on the way */
    unsigned long long mg_sum = 0ull;
    unsigned wmax = 0u;
    if (turn.ok) {
        for (int s = warp; s < ns; s += kWarps) {
            const int v = vid[(32 * s + lane) >> lg], sub = lane & ((1 << lg) - 1), b = soff[s] >> 5, W = soff[s] & 31;
            long long k0 = 0;
            int deg = 0, lo = INT32_MAX, hi = INT32_MIN;
            if (v >= 0) {
                k0 = p.rp[v];
                deg = (int)(p.rp[v + 1] - k0);
            }
            int2 *out = E + 32 * (long long)b + lane;
            for (int j0 = 0; j0 < W; j0 += 8) {
                int2 q[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    /* pads: a lane's last edge again, which changes no min and
                     * spares the walk a look; none where lanes share a vertex,
                     * whose pads are more */
                    const int k = lg ? ((j0 + j) << lg) + sub : max(0, min(j0 + j, deg - 1));
                    q[j] = make_int2(-1, 0);
                    if (j0 + j < W && k < deg) q[j] = make_int2(__ldg(p.succ + k0 + k), __ldg(p.w + k0 + k));
                }
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (q[j].x >= 0) q[j].x = GRID ? __ldcg(number + q[j].x) : number[q[j].x];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (j0 + j >= W) continue;
                    out[32 * (j0 + j)] = q[j];
                    if (q[j].x >= 0) {
                        lo = min(lo, q[j].y);
                        hi = max(hi, q[j].y);
                    }
                }
            }
            for (int o = 1 << lg >> 1; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if (deg > 0) {
                if (lo < 0 && sub == 0) mg_sum += (unsigned long long)(-(long long)lo);
                wmax = max(wmax, max(lo < 0 ? 0u - (unsigned)lo : (unsigned)lo, hi < 0 ? 0u - (unsigned)hi : (unsigned)hi));
            }
        }
        /* the heavy ones a warp each, the cut ones a warp per segment */
        auto copy = [&](int h, int k0, int k1) {
            const long long from = p.rp[vid[V * ns + h]];
            const int2 hd = head[h];
            int2 *const to = (hd.x + (hd.y & INT32_MAX) <= h_smem ? H : H2) + hd.x;
            int lo = INT32_MAX, hi = INT32_MIN;
#pragma unroll 1
            for (int k = k0 + lane; k < k1; k += 256) {
                int2 q[8];
#pragma unroll
                for (int j = 0; j < 8; j++)
                    q[j] = k + 32 * j < k1 ? make_int2(__ldg(p.succ + from + k + 32 * j), __ldg(p.w + from + k + 32 * j))
                                           : make_int2(-1, 0);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (q[j].x >= 0) q[j].x = GRID ? __ldcg(number + q[j].x) : number[q[j].x];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (k + 32 * j >= k1) continue;
                    to[k + 32 * j] = q[j];
                    lo = min(lo, q[j].y);
                    hi = max(hi, q[j].y);
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            wmax = max(wmax, max(lo < 0 ? 0u - (unsigned)lo : (unsigned)lo, hi < 0 ? 0u - (unsigned)hi : (unsigned)hi));
            return lo;
        };
        for (int h = warp; h < nmed; h += kWarps) {
            const int lo = copy(h, 0, head[h].y & INT32_MAX);
            if (lane == 0 && lo < 0) mg_sum += (unsigned long long)(-(long long)lo);
        }
        for (int t = warp; t < hb.tasks; t += kWarps) {
            const int h = nmed + (int)(hb.task[t] & 0xffffu), k0 = (int)(hb.task[t] >> 16) * seg;
            const int lo = copy(h, k0, min(head[h].y & INT32_MAX, k0 + seg));
            if (lane == 0) hb.part[t] = lo;
        }
        __syncthreads();
        for (int h = nmed + tid; h < nh; h += kBlock) {
            const int nt = ((head[h].y & INT32_MAX) + seg - 1) / seg;
            long long lo = 0;
            for (int t = 0; t < nt; t++) lo = min(lo, hb.part[hb.first[h - nmed] + t]);
            mg_sum += (unsigned long long)(-lo);
        }
        __syncthreads();
    }
    wmax = __reduce_max_sync(0xffffffffu, wmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mg_sum += __shfl_xor_sync(0xffffffffu, mg_sum, o);
    if (lane == 0) {
        atomicAdd(&s_sum[0], mg_sum);
        atomicMax(&s_sum[1], (unsigned long long)wmax);
    }
    __syncthreads();
    if (GRID) {
        if (tid == 0 && turn.ok) {
            atomicAdd(&c->mg, s_sum[0]);
            atomicMax(&c->wmax, s_sum[1]);
            turn.ok = round_barrier(p, c, it, (unsigned long long)s_sink, &got);
            s_sink = got != 0ull;
            s_sum[0] = __ldcg(&c->mg);
            s_sum[1] = __ldcg(&c->wmax);
        }
        it++;
        __syncthreads();
    }
    /* 5. the width of the credits, here and in the result */
    const unsigned long long mg = s_sum[0], big = s_sum[1];
    const int out_bits = p.bits == 32 || (p.narrow && mg + big < (unsigned long long)INT32_MAX) ? 32 : 64;
    const bool fits32 = mg + big < (unsigned long long)Lim<int>::top && big <= (unsigned long long)Lim<int>::weight_max;
    SweepState st;
    st.phase = SWEEP_PRIMAL;
    st.left = kFirstPrimal;
    st.primal_len = kSecondPrimal;
    st.dual_len = kFirstDual;
    st.stop = s_sink                                                  ? (int)EG_ERR_INVALID
              : out_bits == 32 && mg > (unsigned long long)INT32_MAX ? (int)EG_ERR_OVERFLOW
                                                                      : 0;
    st.rounds = st.sweeps = 0;
    __syncthreads();
    if (tid < 4) s_sum[tid] = 0ull;
    if (tid == 0) {
        if (!GRID) {
            c->mg = mg;
            c->wmax = big;
        }
        /* potentials count weights 2^nshift-fold: more than n times where
         * that fits */
        const unsigned long long limit =
            fits32 ? (unsigned long long)Lim<int>::weight_max : (unsigned long long)Lim<long long>::weight_max;
        int nshift = 0;
        while (nshift < 20 && (1ll << nshift) <= p.n && (big << (nshift + 1)) <= limit) nshift++;
        r.out_bits = out_bits;
        r.mg = (long long)mg;
        r.scale = 1ll << nshift;
    }
    Count cnt = {0u, 0u, 0u, 0ull, 0ull, 0ull};
    __syncthreads();
    auto run = [&](auto credit, auto kind) {
        using CT = decltype(credit);
        if (GRID && (lg || !ns)) solve<CT, decltype(kind)::value, GRID>(&ps, r, hb, turn, st, it, cnt);
        else solve<CT, decltype(kind)::value, false>(&ps, r, hb, turn, st, it, cnt);
    };
    auto run_kind = [&](auto kind) {
        if (fits32) run(0, kind);
        else run(0ll, kind);
    };
    if (!GRID) run_kind(std::integral_constant<int, KIND_CTA>());
    else if (own_smem && edges_smem) run_kind(std::integral_constant<int, KIND_STAGED>());
    else run_kind(std::integral_constant<int, KIND_GLOBAL>());
    unsigned long long sums[4] = {cnt.raised, cnt.lifts, cnt.edges, cnt.changes};
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sums[k] += __shfl_xor_sync(0xffffffffu, sums[k], o);
        if (lane == 0) atomicAdd(&s_sum[k], sums[k]);
    }
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&c->num_top, s_sum[0]);
        atomicAdd(&c->lifts, s_sum[1]);
        atomicAdd(&c->edges, s_sum[2]);
        atomicAdd(&c->changes, s_sum[3]);
        if (blockIdx.x == 0) {
            c->s = st;
            c->out_bits = out_bits;
        }
    }
}

/* What the kernels may use of a device, asked for once: SMs, and dynamic
 * shared memory per CTA of the one-CTA and the grid kernel (to which they are
 * opted in). */
struct SweepDevice {
    std::atomic<int> sms, smem[2];
};
static SweepDevice g_device[64];

static eg_status sweep_device(int *sms, int *smem)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev >= 64) return eg_set_error(EG_ERR_CUDA, "sweep kernel set-up: %s", cudaGetErrorString(e));
    SweepDevice &d = g_device[dev];
    if (!d.sms.load()) {
        int count = 0, optin = 0;
        e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        for (int k = 0; k < 2; k++) {
            const void *fn = k ? (const void *)k_sweep<true> : (const void *)k_sweep<false>;
            cudaFuncAttributes fa;
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
            if (e == cudaSuccess) d.smem[k] = optin - (int)fa.sharedSizeBytes;
            if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, d.smem[k].load());
        }
        if (e != cudaSuccess) return eg_set_error(EG_ERR_CUDA, "sweep kernel set-up: %s", cudaGetErrorString(e));
        d.sms = count;
    }
    *sms = d.sms;
    smem[0] = d.smem[0];
    smem[1] = d.smem[1];
    return EG_OK;
}

eg_status sweep_plan(int n, long long m, int max_ctas, SweepPlan *plan)
{
    int sms = 0, smem_of[2];
    eg_status s = sweep_device(&sms, smem_of);
    if (s != EG_OK) return s;
    const long long total = 8 * m + m / 2 + (long long)kVertexBytes * n;
    memset(plan, 0, sizeof *plan);
    plan->block = kBlock;
    plan->grid = 1;
    if (total + kSlackBytes <= smem_of[0]) {
        plan->one_cta = 1;
        plan->smem_bytes = (int)(total + kSlackBytes);
        return EG_OK;
    }
    const int bytes = smem_of[1];
    plan->grid = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
    plan->smem_bytes = bytes;
    plan->values = (size_t)n + (size_t)kPadSlots * plan->grid;
    /* a part that ends with a vertex of many edges may not fit shared memory
     * even where the mean part does */
    plan->edges = (size_t)(m + m / 16) + (size_t)kPadEdges * plan->grid;
    if (total / plan->grid + kSlackBytes > bytes) {
        plan->vids = plan->values;
        plan->offs = plan->values / 32 + 4 * (size_t)plan->grid + 4;
    }
    return EG_OK;
}

eg_status launch_sweep(SweepParams p, const SweepPlan &plan, cudaStream_t st)
{
    p.smem_bytes = plan.smem_bytes;
    void *args[] = {(void *)&p};
    cudaError_t e;
    if (plan.one_cta)
        e = cudaLaunchKernel((const void *)k_sweep<false>, dim3(1), dim3(kBlock), args, (size_t)plan.smem_bytes, st);
    else
        e = cudaLaunchCooperativeKernel((const void *)k_sweep<true>, dim3(plan.grid), dim3(kBlock), args,
                                        (size_t)plan.smem_bytes, st);
    if (e != cudaSuccess) return eg_set_error(EG_ERR_CUDA, "launch of the sweep kernel failed: %s", cudaGetErrorString(e));
    return EG_OK;
}

}  // namespace eg
