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
 * Schedule (advanced by each round's last arriver, on the device):
 *   primal   sweeps of credit lifts; a round without a raise ends the solve;
 *   dual     sweeps that raise D, without a barrier between them, then a
 *            copy K = D;
 *   kill     sweeps that set K(u) = out where u's condition fails on K, until
 *            a round removes nothing: what is left is the largest S.  Its
 *            credits become TOP;
 *   primal   again, longer, and so on with longer dual phases.
 * A lift of every credit reads values that are initial, raised or certified,
 * all at most the least fixed point, and a primal round without a raise and
 * without a newly certified vertex has lifted every vertex against the final
 * credits: the result is the least fixed point, as of any fair schedule.
 *
 * Layout.  The grid kernel runs one 1024-thread CTA per SM.  A CTA owns a
 * contiguous vertex range, cut so that 8 B per edge + 28 B per vertex is the
 * same for all; it keeps its vertices' credits and potentials, row offsets
 * and (when they fit) edges in shared memory for the whole solve, so a sweep
 * reads only the successors' values from L2.  `lanes` lanes share a vertex
 * (the mean out-degree rounded down to a power of two); vertices with more
 * out-edges than kHubEdges are cut into segments dealt to the CTA's warps.
 * Nothing is renumbered and no transpose is needed.  A game of at most
 * sweep_cta_bytes() <= the shared memory of a CTA runs in one CTA, with every
 * value in shared memory and __syncthreads for a barrier.
 *
 * What bounds it: the chain of a sweep (shared-memory edge, L2 gather, store,
 * barrier) on small games, one gather per clock and SM on large ones.
 * Measured, whole solve on the device, against the frontier and dense rounds
 * that climb to MG: random 2..16-regular game of 131,072 vertices 684 ms ->
 * 0.43 ms (16 primal sweeps for 40,000), of 16,000 vertices 82 ms -> 0.18 ms;
 * power-law game of 2^20 vertices and 8.3 M edges 9.3 s -> 16 ms; complete
 * digraph of 2,000 vertices 14.2 ms -> 0.49 ms; 4-regular game of 1,000
 * vertices (one CTA) 4.1 ms -> 0.11 ms.
 *
 * Credits are int64 with TOP = 2^62 while the solve runs: OMINUS(a, w) is
 * g(a - w) with g(x) = x > MG ? TOP : max(x, 0), and MG + max |w| < 2^62
 * for every game that fits the 32-bit sizes, so a TOP successor always gives
 * TOP; g is monotone and is applied once, after the min or max.
 */
#include "eg_sweep.cuh"

#include <algorithm>

namespace eg {

constexpr int kSweepBlock = 1024;
constexpr int kHubEdges = 256;  /* out-edges above which a vertex is cut      */
constexpr int kMaxTasks = 1040; /* segments of a CTA's cut vertices           */
constexpr int kMaxHubs = 520;
constexpr int kVertexBytes = 28; /* row offset, credit, potential, its copy   */
constexpr int kFirstPrimal = 4, kFirstDual = 8, kSecondPrimal = 16, kMaxDual = 32, kMaxPrimal = 1 << 16;
constexpr int kKillSweeps = 2;   /* kill sweeps between two grid barriers     */

constexpr long long kTop = 1LL << 62;    /* credit TOP; potential "out of S"  */
constexpr long long kLow = -(1LL << 62); /* potential of a vertex at TOP      */
constexpr long long kDualMax = 1LL << 61;

/* What a CTA knows of its vertex range. */
struct Range {
    int va, nv;              /* vertices [va, va + nv)                       */
    int ne;                  /* their edges                                  */
    const unsigned *off;     /* shared: first edge | owner << 31; or null    */
    const long long *rp;     /* global row offsets of the range              */
    long long e0;
    const int2 *Es;          /* the edges in shared memory, or null          */
    const int *succ, *w;     /* global, at the range's first edge            */
    const unsigned char *owner;
    int n0;
    long long *myF, *myD, *myK; /* own values (shared, or global at va)      */
    long long *gF, *gD, *gK; /* grid: the global values at va, which gathers read */
    int lanes, nshift;
    __device__ __forceinline__ void vertex(int i, int &b, int &e, bool &own) const
    {
        if (off) {
            const unsigned x = off[i];
            b = (int)(x & 0x7fffffffu);
            e = (int)(off[i + 1] & 0x7fffffffu);
            own = (x >> 31) != 0u;
        } else {
            b = (int)(rp[i] - e0);
            e = (int)(rp[i + 1] - e0);
            own = owner ? owner[va + i] != 0 : va + i >= n0;
        }
    }
};

struct Hubs {
    int count, tasks, seg;
    int hub[kMaxHubs], first[kMaxHubs]; /* vertex index; its first segment    */
    unsigned task[kMaxTasks];           /* hub | segment << 16                */
    long long part[kMaxTasks];
};

struct SweepCount {
    unsigned raised, lifts;
    unsigned long long edges;
};

enum { MODE_PRIMAL, MODE_DUAL, MODE_KILL, MODE_SETUP };

__device__ __forceinline__ long long shfl_xor_ll(long long v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }

/* Values read by gathers: other SMs write them (grid), or shared memory. */
template <bool GRID>
__device__ __forceinline__ long long gather(const long long *p)
{
    return GRID ? __ldcg(p) : *p;
}

/* One edge's value in "min space": the lane keeps the least.  A max is the
 * min of negated values. */
template <int MODE>
__device__ __forceinline__ long long edge_value(long long x, int w, bool own, int nshift)
{
    if (MODE == MODE_PRIMAL) {
        const long long v = x - (long long)w;
        return own ? -v : v;
    }
    const long long v = x + ((long long)w << nshift) + 1;
    return own ? v : -v;
}

template <bool GRID, bool ES, int MODE>
__device__ __forceinline__ long long walk_edges(const Range &r, const long long *G, int k, int e, int step, bool own,
                                                int nshift)
{
    long long acc = INT64_MAX;
    for (; k < e; k += 2 * step) {
        const bool two = k + step < e;
        int s0, w0, s1 = 0, w1 = 0;
        if (ES) {
            const int2 q = r.Es[k];
            s0 = q.x;
            w0 = q.y;
            if (two) {
                const int2 t = r.Es[k + step];
                s1 = t.x;
                w1 = t.y;
            }
        } else {
            s0 = MODE == MODE_SETUP ? 0 : __ldg(r.succ + k);
            w0 = __ldg(r.w + k);
            if (two) {
                s1 = MODE == MODE_SETUP ? 0 : __ldg(r.succ + k + step);
                w1 = __ldg(r.w + k + step);
            }
        }
        if (MODE == MODE_SETUP) { /* the least weight; largest |weight| in the high part is kept by the caller */
            acc = min(acc, (long long)w0);
            if (two) acc = min(acc, (long long)w1);
        } else {
            const long long x0 = gather<GRID>(G + s0);
            const long long x1 = two ? gather<GRID>(G + s1) : 0;
            acc = min(acc, edge_value<MODE>(x0, w0, own, nshift));
            if (two) acc = min(acc, edge_value<MODE>(x1, w1, own, nshift));
        }
    }
    return acc;
}

/* The vertex's own value, and whether this kind of sweep passes it over. */
template <int MODE>
__device__ __forceinline__ bool own_value(const Range &r, int i, long long &old)
{
    if (MODE == MODE_SETUP) return true;
    old = MODE == MODE_PRIMAL ? r.myF[i] : MODE == MODE_DUAL ? r.myD[i] : r.myK[i];
    return old < kTop && old != kLow;
}

/* The last step of a vertex (one lane): acc is the min-space result. */
template <bool GRID, int MODE>
__device__ __forceinline__ void finish_vertex(const Range &r, int i, bool own, long long old,
                                              long long acc, int deg, long long mg, unsigned long long &mg_sum,
                                              SweepCount &cnt)
{
    if (MODE == MODE_SETUP) {
        if (acc < 0) mg_sum += (unsigned long long)(-acc);
        return;
    }
    if (MODE == MODE_PRIMAL) {
        const long long x = own ? -acc : acc;
        const long long nv = x > mg ? kTop : (x > 0 ? x : 0);
        cnt.lifts++;
        cnt.edges += (unsigned)deg;
        if (nv > old) {
            cnt.raised++;
            r.myF[i] = nv;
            if (GRID) __stcg(r.gF + i, nv);
            if (nv == kTop) {
                r.myD[i] = kLow;
                if (GRID) __stcg(r.gD + i, kLow);
            }
        }
        return;
    }
    long long y = own ? acc : -acc;
    y = y > 0 ? y : 0;
    if (y <= old) return;
    if (MODE == MODE_DUAL) {
        if (y > kDualMax) y = kTop;
        r.myD[i] = y;
        if (GRID) __stcg(r.gD + i, y);
    } else {
        cnt.raised++;
        r.myK[i] = kTop;
        if (GRID) __stcg(r.gK + i, kTop);
    }
}

/* One sweep of the CTA's vertices. */
template <bool GRID, bool ES, int MODE>
__device__ __forceinline__ void sweep(const Range &range, Hubs &hb, const long long *G, long long mg,
                                   unsigned long long &mg_out, SweepCount &cnt_out)
{
    /* copies in registers: stores to credits cannot alias them */
    const Range r = range;
    SweepCount cnt = cnt_out;
    unsigned long long mg_sum = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int nwarps = kSweepBlock / 32;
    const int g = r.lanes, gl = lane & (g - 1);
    const int nshift = r.nshift;
    const bool hubs = hb.count > 0;
    if (hubs) {
        for (int t = warp; t < hb.tasks; t += nwarps) {
            const unsigned tk = hb.task[t];
            const int i = hb.hub[tk & 0xffffu];
            int b, e;
            bool own;
            long long old = 0;
            r.vertex(i, b, e, own);
            long long acc = INT64_MAX;
            if (own_value<MODE>(r, i, old)) {
                const int k0 = b + (int)(tk >> 16) * hb.seg;
                acc = walk_edges<GRID, ES, MODE>(r, G, k0 + lane, min(e, k0 + hb.seg), 32, own, nshift);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc = min(acc, shfl_xor_ll(acc, o));
            if (lane == 0) hb.part[t] = acc;
        }
    }
    const int per = 32 / g;
    for (int i0 = warp * per; i0 < r.nv; i0 += nwarps * per) {
        const int i = i0 + lane / g;
        int b = 0, e = 0;
        bool own = false;
        long long old = 0;
        bool act = i < r.nv;
        if (act) {
            r.vertex(i, b, e, own);
            act = (e - b <= hb.seg || !hubs) && own_value<MODE>(r, i, old);
        }
        long long acc = INT64_MAX;
        if (act) acc = walk_edges<GRID, ES, MODE>(r, G, b + gl, e, g, own, nshift);
        __syncwarp();
        for (int o = g >> 1; o > 0; o >>= 1) acc = min(acc, shfl_xor_ll(acc, o));
        if (act && gl == 0) finish_vertex<GRID, MODE>(r, i, own, old, acc, e - b, mg, mg_sum, cnt);
    }
    if (hubs) {
        __syncthreads();
        for (int h = warp; h < hb.count; h += nwarps) {
            const int i = hb.hub[h];
            int b, e;
            bool own;
            long long old = 0;
            r.vertex(i, b, e, own);
            const int nt = (e - b + hb.seg - 1) / hb.seg;
            long long acc = INT64_MAX;
            for (int t = lane; t < nt; t += 32) acc = min(acc, hb.part[hb.first[h] + t]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc = min(acc, shfl_xor_ll(acc, o));
            if (lane == 0 && own_value<MODE>(r, i, old))
                finish_vertex<GRID, MODE>(r, i, own, old, acc, e - b, mg, mg_sum, cnt);
        }
        __syncthreads();
    }
    cnt_out = cnt;
    if (MODE == MODE_SETUP) mg_out += mg_sum;
}

/* The schedule after a round in which `raised` values changed. */
__device__ __forceinline__ void advance(const SweepParams &p, SweepCtrl *c, int ran, unsigned long long raised)
{
    if (c->phase == SWEEP_PRIMAL) {
        const long long round = c->rounds;
        c->rounds = round + 1;
        c->sweeps += ran;
        c->left -= ran;
        c->changes += raised;
        if (raised == 0ull) {
            c->phase = SWEEP_DONE;
            return;
        }
        if (p.max_rounds >= 0 && round + 1 >= p.max_rounds) c->stop = (int)EG_ERR_LOOPCAP;
        else if (p.timeout_ns && globaltimer_ns() - c->t_start > p.timeout_ns) c->stop = (int)EG_ERR_TIMEOUT;
        else if (p.cancel && (round & 63) == 0 && ld_volatile(p.cancel)) c->stop = (int)EG_ERR_CANCELLED;
        if (c->stop) return;
        if (c->left <= 0) {
            if (p.hand_sweeps && c->sweeps >= p.hand_sweeps && (long long)raised < p.hand_raised) {
                c->phase = SWEEP_HANDOVER;
                return;
            }
            c->phase = SWEEP_DUAL;
            c->left = c->dual_len;
        }
    } else if (c->phase == SWEEP_DUAL) {
        c->dual_sweeps += ran;
        c->dual_len = min(2 * c->dual_len, kMaxDual);
        c->phase = SWEEP_KILL;
    } else {
        c->kill_sweeps += ran;
        if (raised == 0ull) {
            c->attempts++;
            c->phase = SWEEP_PRIMAL;
            c->left = c->primal_len;
            c->primal_len = min(2 * c->primal_len, kMaxPrimal);
        }
    }
}

/* First vertex v with 8 rp[v] + 28 v >= target, for two targets at once: a
 * search in which every thread probes one place per step. */
__device__ __forceinline__ void find_range(const SweepParams &p, unsigned long long ta, unsigned long long tb, int &va,
                                           int &vb)
{
    constexpr int half = kSweepBlock / 2;
    const bool first = threadIdx.x < half;
    const int t = threadIdx.x & (half - 1);
    const unsigned long long target = first ? ta : tb;
    int lo[2] = {0, 0}, hi[2] = {p.n, p.n}; /* the answer is in [lo, hi] */
    while (lo[0] < hi[0] || lo[1] < hi[1]) {
        const int l = first ? lo[0] : lo[1], h = first ? hi[0] : hi[1];
        const int step = (h - l + half - 1) / half;
        const long long at = (long long)l + (long long)t * step;
        const bool below = at < h && (unsigned long long)p.rp[at] * 8ull + (unsigned long long)at * kVertexBytes < target;
        const int ca = __syncthreads_count(below && first);
        const int cb = __syncthreads_count(below && !first);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int c = k ? cb : ca;
            const int l2 = lo[k], h2 = hi[k];
            if (l2 >= h2) continue;
            const int st = (h2 - l2 + half - 1) / half;
            const long long next = (long long)l2 + (long long)c * st; /* first probe not below */
            if (c > 0) lo[k] = (int)(l2 + (long long)(c - 1) * st + 1);
            if (next < h2) hi[k] = (int)next;
        }
    }
    va = lo[0];
    vb = lo[1];
}

template <bool GRID>
__global__ void __launch_bounds__(kSweepBlock, 1) k_sweep(const __grid_constant__ SweepParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Hubs hb;
    __shared__ unsigned long long s_sum[4];
    __shared__ SweepCtrl s_ctrl; /* one-CTA kernel */
    SweepCtrl *c = GRID ? p.ctrl : &s_ctrl;
    const int tid = threadIdx.x, lane = tid & 31;
    if (!GRID) {
        for (int i = tid; i < (int)(sizeof(SweepCtrl) / 4); i += kSweepBlock) ((int *)&s_ctrl)[i] = 0;
        __syncthreads();
    }
    if (tid == 0 && blockIdx.x == 0) c->t_start = globaltimer_ns();
    Range r;
    int vb;
    if (GRID) {
        const unsigned long long total = (unsigned long long)p.m * 8ull + (unsigned long long)p.n * kVertexBytes;
        const unsigned long long g = gridDim.x, b = blockIdx.x;
        find_range(p, total / g * b + total % g * b / g, total / g * (b + 1) + total % g * (b + 1) / g, r.va, vb);
        if (b + 1 == g) vb = p.n;
    } else {
        r.va = 0;
        vb = p.n;
    }
    r.nv = vb - r.va;
    r.e0 = p.rp[r.va];
    r.ne = (int)(p.rp[vb] - r.e0);
    r.rp = p.rp + r.va;
    r.succ = p.succ + r.e0;
    r.w = p.w + r.e0;
    r.owner = p.owner;
    r.n0 = p.n0;
    r.gF = p.F + r.va;
    r.gD = p.D + r.va;
    r.gK = p.K + r.va;
    r.lanes = p.lanes;
    r.nshift = p.nshift;
    /* shared memory: own values and row offsets, then the edges */
    const long long own_bytes = ((long long)r.nv * kVertexBytes + 4 + 15) & ~15LL;
    const bool own_fits = own_bytes <= p.smem_bytes;
    r.off = nullptr;
    r.Es = nullptr;
    if (own_fits) {
        r.myF = (long long *)smem;
        r.myD = r.myF + r.nv;
        r.myK = r.myD + r.nv;
        unsigned *off = (unsigned *)(r.myK + r.nv);
        r.off = off;
        for (int i = tid; i <= r.nv; i += kSweepBlock) {
            unsigned own = 0;
            if (i < r.nv) own = p.owner ? (unsigned)(p.owner[r.va + i] != 0) : (unsigned)(r.va + i >= p.n0);
            off[i] = (unsigned)(r.rp[i] - r.e0) | own << 31;
        }
        if (own_bytes + 8LL * r.ne <= p.smem_bytes) {
            int2 *Es = (int2 *)(smem + own_bytes);
            r.Es = Es;
            for (int k = tid; k < r.ne; k += kSweepBlock) Es[k] = make_int2(__ldg(r.succ + k), __ldg(r.w + k));
        }
    } else {
        r.myF = r.gF;
        r.myD = r.gD;
        r.myK = r.gK;
    }
    for (int i = tid; i < r.nv; i += kSweepBlock) {
        r.myF[i] = 0;
        r.myD[i] = 0;
        if (GRID && own_fits) {
            __stcg(r.gF + i, 0LL);
            __stcg(r.gD + i, 0LL);
        }
    }
    /* the range's heavy vertices, cut into at most kMaxTasks segments */
    const int seg = max(kHubEdges, (r.ne / 512 + 31) & ~31);
    if (tid == 0) {
        hb.count = 0;
        hb.tasks = 0;
        hb.seg = seg;
    }
    if (tid < 4) s_sum[tid] = 0ull;
    __syncthreads();
    for (int i = tid; i < r.nv; i += kSweepBlock) {
        int b, e;
        bool own;
        r.vertex(i, b, e, own);
        if (e - b > seg) {
            const int h = atomicAdd(&hb.count, 1);
            const int nt = (e - b + seg - 1) / seg;
            const int t0 = atomicAdd(&hb.tasks, nt);
            hb.hub[h] = i;
            hb.first[h] = t0;
            for (int t = 0; t < nt; t++) hb.task[t0 + t] = (unsigned)h | (unsigned)t << 16;
        }
    }
    __syncthreads();
    /* MG and the largest |weight| */
    SweepCount cnt = {0u, 0u, 0ull};
    unsigned long long mg_sum = 0;
    if (r.Es) sweep<GRID, true, MODE_SETUP>(r, hb, nullptr, 0, mg_sum, cnt);
    else sweep<GRID, false, MODE_SETUP>(r, hb, nullptr, 0, mg_sum, cnt);
    unsigned wmax = 0;
    for (int k = tid; k < r.ne; k += kSweepBlock) {
        const int x = r.Es ? r.Es[k].y : __ldg(r.w + k);
        wmax = max(wmax, (unsigned)(x < 0 ? -(long long)x : (long long)x));
    }
    wmax = __reduce_max_sync(0xffffffffu, wmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mg_sum += __shfl_xor_sync(0xffffffffu, mg_sum, o);
    if (lane == 0) {
        atomicAdd(&s_sum[0], mg_sum);
        atomicMax(&s_sum[1], (unsigned long long)wmax);
    }
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&c->mg, s_sum[0]);
        atomicMax(&c->wmax, s_sum[1]);
    }
    auto first = [&]() {
        const bool fast32 = c->mg + c->wmax < (unsigned long long)INT32_MAX;
        c->out_bits = p.bits == 32 || (p.narrow && fast32) ? 32 : 64;
        if (c->out_bits == 32 && c->mg > (unsigned long long)INT32_MAX) c->stop = (int)EG_ERR_OVERFLOW;
        c->phase = SWEEP_PRIMAL;
        c->left = kFirstPrimal;
        c->primal_len = kSecondPrimal;
        c->dual_len = kFirstDual;
    };
    bool ok = true;
    if (GRID) {
        ok = grid_barrier(c, p.wait_limit_ns, first);
    } else {
        __syncthreads();
        if (tid == 0) first();
        __syncthreads();
    }
    const long long mg = (long long)ld_volatile_u64(&c->mg);
    /* values that gathers read: own arrays of the one CTA, or the global ones */
    const long long *GF = GRID ? p.F : r.myF, *GD = GRID ? p.D : r.myD, *GK = GRID ? p.K : r.myK;
    unsigned certified = 0;
    int phase = SWEEP_PRIMAL;
    for (unsigned it = 0; ok && !ld_volatile(&c->stop); it++) {
        const int was = phase;
        phase = ld_volatile(&c->phase);
        if (phase == SWEEP_DONE || phase == SWEEP_HANDOVER) break;
        const int left = ld_volatile(&c->left);
        const unsigned raised0 = cnt.raised;
        int ran;
        if (phase == SWEEP_PRIMAL) {
            if (was == SWEEP_KILL) {
                /* the certified vertices: TOP */
                for (int i = tid; i < r.nv; i += kSweepBlock) {
                    const long long k = r.myK[i];
                    if (k < kTop && k != kLow) {
                        r.myF[i] = kTop;
                        r.myD[i] = kLow;
                        if (GRID) {
                            __stcg(r.gF + i, kTop);
                            __stcg(r.gD + i, kLow);
                        }
                        cnt.raised++;
                        certified++;
                    }
                }
                __syncthreads();
            }
            ran = GRID ? min(p.sweeps, left) : 1;
            for (int s = 0; s < ran; s++) {
                if (r.Es) sweep<GRID, true, MODE_PRIMAL>(r, hb, GF, mg, mg_sum, cnt);
                else sweep<GRID, false, MODE_PRIMAL>(r, hb, GF, mg, mg_sum, cnt);
            }
        } else if (phase == SWEEP_DUAL) {
            ran = left;
            for (int s = 0; s < ran; s++) {
                if (r.Es) sweep<GRID, true, MODE_DUAL>(r, hb, GD, mg, mg_sum, cnt);
                else sweep<GRID, false, MODE_DUAL>(r, hb, GD, mg, mg_sum, cnt);
            }
            __syncthreads();
            for (int i = tid; i < r.nv; i += kSweepBlock) {
                const long long d = r.myD[i];
                r.myK[i] = d;
                if (GRID) __stcg(r.gK + i, d);
            }
        } else {
            ran = GRID ? kKillSweeps : 1;
            for (int s = 0; s < ran; s++) {
                if (r.Es) sweep<GRID, true, MODE_KILL>(r, hb, GK, mg, mg_sum, cnt);
                else sweep<GRID, false, MODE_KILL>(r, hb, GK, mg, mg_sum, cnt);
            }
        }
        const unsigned d = __reduce_add_sync(0xffffffffu, cnt.raised - raised0);
        if (GRID) {
            if (tid == 0) s_sum[2] = 0ull;
            __syncthreads();
            if (lane == 0 && d) atomicAdd(&s_sum[2], (unsigned long long)d);
            __syncthreads();
            if (tid == 0 && s_sum[2]) atomicAdd(&c->raised[it & 1], s_sum[2]);
            ok = grid_barrier(c, p.wait_limit_ns, [&]() {
                const unsigned long long raised = c->raised[it & 1];
                c->raised[(it + 1) & 1] = 0ull;
                advance(p, c, ran, raised);
            });
        } else {
            if (lane == 0 && d) atomicAdd(&c->raised[it & 1], (unsigned long long)d);
            __syncthreads();
            if (tid == 0) {
                const unsigned long long raised = c->raised[it & 1];
                c->raised[(it + 1) & 1] = 0ull;
                advance(p, c, ran, raised);
            }
            __syncthreads();
        }
    }
    __syncthreads();
    /* credits out */
    const int out_bits = ld_volatile(&c->out_bits);
    unsigned tops = 0;
    for (int i = tid; i < r.nv; i += kSweepBlock) {
        const long long f = r.myF[i];
        tops += f == kTop;
        if (out_bits == 32) ((int *)p.out)[r.va + i] = f == kTop ? INT32_MAX : (int)f;
        else ((long long *)p.out)[r.va + i] = f == kTop ? (long long)INT64_MAX : f;
    }
    tops = __reduce_add_sync(0xffffffffu, tops);
    certified = __reduce_add_sync(0xffffffffu, certified);
    const unsigned lifts = __reduce_add_sync(0xffffffffu, cnt.lifts);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt.edges += __shfl_xor_sync(0xffffffffu, cnt.edges, o);
    if (tid < 4) s_sum[tid] = 0ull;
    __syncthreads();
    if (lane == 0) {
        atomicAdd(&s_sum[0], (unsigned long long)tops);
        atomicAdd(&s_sum[1], (unsigned long long)certified);
        atomicAdd(&s_sum[2], (unsigned long long)lifts);
        atomicAdd(&s_sum[3], cnt.edges);
    }
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&c->num_top, s_sum[0]);
        atomicAdd(&c->certified, s_sum[1]);
        atomicAdd(&c->lifts, s_sum[2]);
        atomicAdd(&c->edges, s_sum[3]);
    }
    if (!GRID) {
        __syncthreads();
        for (int i = tid; i < (int)(sizeof(SweepCtrl) / 4); i += kSweepBlock) ((int *)p.ctrl)[i] = ((int *)&s_ctrl)[i];
    }
}

long long sweep_cta_bytes(long long n, long long m)
{
    return ((n * kVertexBytes + 4 + 15) & ~15LL) + 8 * m;
}

/* Dynamic shared memory a CTA of the kernel may have. */
static eg_status sweep_smem(const void *fn, int dev, int *bytes)
{
    int optin = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return eg_set_error(EG_ERR_CUDA, "sweep kernel attributes: %s", cudaGetErrorString(e));
    *bytes = optin - (int)fa.sharedSizeBytes;
    return EG_OK;
}

eg_status launch_sweep(SweepParams p, cudaStream_t st, int max_ctas, int *grid, int *block)
{
    const void *one = (const void *)k_sweep<false>, *all = (const void *)k_sweep<true>;
    int dev = 0, sms = 0, bytes = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return eg_set_error(EG_ERR_CUDA, "sweep kernel set-up: %s", cudaGetErrorString(e));
    *block = kSweepBlock;
    const long long need = sweep_cta_bytes(p.n, p.m);
    eg_status s = sweep_smem(one, dev, &bytes);
    if (s != EG_OK) return s;
    if (need <= bytes) {
        *grid = 1;
        p.smem_bytes = (int)need;
        e = cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        void *args[] = {(void *)&p};
        if (e == cudaSuccess) e = cudaLaunchKernel(one, dim3(1), dim3(kSweepBlock), args, (size_t)need, st);
    } else {
        s = sweep_smem(all, dev, &bytes);
        if (s != EG_OK) return s;
        *grid = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
        p.smem_bytes = bytes;
        e = cudaFuncSetAttribute(all, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        void *args[] = {(void *)&p};
        if (e == cudaSuccess)
            e = cudaLaunchCooperativeKernel(all, dim3(*grid), dim3(kSweepBlock), args, (size_t)bytes, st);
    }
    if (e != cudaSuccess) return eg_set_error(EG_ERR_CUDA, "launch of the sweep kernel failed: %s", cudaGetErrorString(e));
    return EG_OK;
}

}  // namespace eg
