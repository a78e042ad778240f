/*
 * eg_serve.cu -- serving mean-payoff threshold queries with continuous
 * batching.
 *
 * A query asks for the credits of every vertex of a registered game at K
 * thresholds p_k (weights w*d - p_k).  One worker thread runs the loop:
 *
 *   1. completions: micro-batches whose event fired hand their credits to
 *      their queries (device -> host) and release the queries' buffers;
 *   2. admission, in submission order: a query is admitted when fewer than
 *      max_inflight queries are admitted and the free device memory (from
 *      cudaMemGetInfo and what the pool holds idle, less what queries admitted
 *      since that look take) minus hbm_reserve_bytes covers its credits and,
 *      if its game is not resident yet, the game's packed layout; idle
 *      resident games are evicted oldest-first when memory is short.  A game
 *      stays resident across all its queries until it is evicted or removed;
 *   3. launch: the admitted queries not yet launched go into one or two
 *      micro-batches, i.e. launches of the unit kernels (eg_batch.cu: one CTA
 *      per game x threshold group, credits in shared memory), each on the next
 *      of `streams` streams.  A micro-batch some of whose units went to the
 *      cluster tail gets its tail launched when its units have ended.
 *      Earlier micro-batches keep running; as their CTAs run out of units and
 *      exit, the new launch's CTAs take the freed SMs, so the work of queries
 *      that arrived at different times overlaps on the device.  Each launch records its first CTA start and last CTA end
 *      on the device clock (eg_serve_trace).
 *
 * Routing: games above the batched layout's limit (2^19 vertices), and games
 * whose credits do not fit one CTA's shared memory while the queue is
 * shallow, are solved by a second thread one threshold at a time on the
 * persistent grid solver, capped at `large_ctas` CTAs so that micro-batches
 * keep SMs to run on: a CTA of it fills an SM, so by default it gets three
 * quarters of them (on all, a query of 2,000 vertices waited 50 s for the end
 * of a path of 600,000).  With a deep queue such games run as units with their
 * credits in global memory, for throughput.
 *
 * Every result equals the solve of the same game and threshold alone: a
 * unit's work depends only on its own game and thresholds.
 */
#include "eg_batch.cuh"
#include "eg_pool.cuh"
#include "../../include/egsolver_b200_serve.h"

#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

using namespace eg;

namespace {

using clk = std::chrono::steady_clock;

double ms_since(clk::time_point a, clk::time_point b) { return std::chrono::duration<double, std::milli>(b - a).count(); }

struct ServedGame {
    int64_t id;
    int n, n0;
    long long m;
    std::vector<int64_t> rp;
    std::vector<int32_t> succ, w;
    std::vector<uint8_t> own;
    bool has_owner = false;
    bool large = false;          /* above the batched layout's limit         */
    bool fits_smem = true;       /* one threshold's credits fit shared memory */
    bool resident = false;
    bool removed = false;
    HostPacked hp;               /* packed layout (host image)               */
    PackedDev pd;                /* its device copy while resident           */
    int active = 0; /* admitted queries still running */
    uint64_t last_use = 0;
    eg_game view() const
    {
        eg_game g;
        g.num_nodes = n;
        g.num_nodes0 = n0;
        g.num_edges = m;
        g.row_ptr = rp.data();
        g.succ = succ.data();
        g.weight = w.data();
        g.owner = has_owner ? own.data() : nullptr;
        return g;
    }
};

struct Query {
    int64_t id, game;
    int K, d;
    std::vector<int> p;
    int state = EG_QUERY_QUEUED;
    eg_status status = EG_OK;
    clk::time_point t_submit, t_done;
    long long rounds = 0;
    std::unique_ptr<int64_t[]> result; /* threshold-major, n * K */
    size_t result_len = 0;
    std::vector<long long> mg;   /* MG per threshold                         */
    /* device buffers while admitted: credits n*K (threshold-major),
     * thresholds, MG, per-unit rounds and status, global credit scratch */
    long long *dF = nullptr;
    int *dthr = nullptr;
    long long *dmg = nullptr;
    long long *drounds = nullptr;
    int *dstatus = nullptr;
    void *dscratch = nullptr;
    size_t dbytes = 0, o_rounds = 0, o_status = 0, o_end = 0; /* places in the block */
    std::vector<UnitDesc> units; /* planned at admission                     */
    std::vector<long long> cost;
    int smem = 16;
    cudaEvent_t ready = nullptr; /* buffers allocated and thresholds copied */
};

struct Launch {
    int stream;
    int64_t number = 0;
    int units = 0;
    Lane *lane = nullptr;       /* its first event: the end; its page: the control block by then */
    std::vector<int64_t> qids;
    void *block = nullptr;      /* device memory of what follows              */
    UnitDesc *dunits = nullptr;
    LaunchCtrl *dctrl = nullptr;
    TailList *tl = nullptr;
    void *dscratch = nullptr;   /* hybrid tail regions                        */
    UnitSet set;                /* for the tail's launch                      */
    bool in_tail = false;       /* the tail's kernels are launched            */
};

}  // namespace

struct eg_server {
    eg_serve_opts o;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::thread worker, large_worker;
    bool stop = false;
    int64_t next_game = 1, next_query = 1;
    std::map<int64_t, std::unique_ptr<ServedGame>> games;
    std::map<int64_t, std::unique_ptr<Query>> queries;
    std::deque<int64_t> pending, large_pending;
    std::vector<int64_t> ready;
    std::vector<Launch> inflight;
    std::vector<cudaStream_t> streams;
    std::vector<UnitLauncher> launchers; /* side streams of each micro-batch stream */
    cudaStream_t upload_stream = nullptr;
    int next_stream = 0;
    int admitted_now = 0;
    uint64_t tick = 0;
    int sms = 148;
    int smem_budget = 0;
    std::vector<eg_serve_span> spans;   /* device-clock span of every micro-batch */
    unsigned long long clock0 = 0;      /* device clock of the first micro-batch  */
    /* statistics */
    int64_t submitted = 0, admitted = 0, completed = 0, failed = 0, uploads = 0, evictions = 0;
    int64_t micro_batches = 0, threshold_solves = 0;
    std::vector<double> latencies;
    clk::time_point t0, t_last_done;
    int64_t device_bytes = 0;
};

namespace {

/* credits | thresholds | MG | per-unit rounds | per-unit status | scratch */
size_t query_bytes(const ServedGame &g, int K, size_t scratch)
{
    return sizeof(long long) * (size_t)g.n * K + 4 * 64 * sizeof(long long) + 1024 + scratch;
}

void free_query_device(Query &q, cudaStream_t st)
{
    pool_free(q.dF, st);
    if (q.ready) cudaEventDestroy(q.ready);
    q.ready = nullptr;
    q.dF = nullptr;
    q.dthr = nullptr;
    q.dmg = nullptr;
    q.drounds = nullptr;
    q.dstatus = nullptr;
    q.dscratch = nullptr;
}

void drop_resident(eg_server *s, ServedGame &g)
{
    s->device_bytes -= (int64_t)g.pd.bytes;
    pool_free(g.pd.block, s->upload_stream);
    cudaStreamSynchronize(s->upload_stream);
    g.pd = PackedDev();
    g.resident = false;
}

/* Drops the resident game that nobody uses and that was used longest ago. */
bool evict_one(eg_server *s)
{
    ServedGame *victim = nullptr;
    for (auto &kv : s->games) {
        ServedGame &g = *kv.second;
        if (g.resident && g.active == 0 && (!victim || g.last_use < victim->last_use)) victim = &g;
    }
    if (!victim) return false;
    drop_resident(s, *victim);
    s->evictions++;
    return true;
}

/* Makes room for `need` bytes above the reserve.  *left is what the last look
 * found, less what was taken since: a look takes 65 us, most of an admission,
 * and one serves the queries that are admitted together. */
bool make_room(eg_server *s, std::unique_lock<std::mutex> &lk, size_t need, size_t *left)
{
    while (*left < need) {
        size_t free_b = 0, total_b = 0;
        lk.unlock();
        const cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
        free_b += pool_idle(s->o.device);
        lk.lock();
        if (e != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        const size_t reserve = (size_t)s->o.hbm_reserve_bytes;
        *left = free_b > reserve ? free_b - reserve : 0;
        if (*left < need && !evict_one(s)) return false;
        if (*left < need) *left = 0;
    }
    *left -= need;
    return true;
}

void finish_query(eg_server *s, Query &q, eg_status st, clk::time_point now)
{
    q.status = st;
    q.state = st == EG_OK ? EG_QUERY_DONE : EG_QUERY_FAILED;
    q.t_done = now;
    s->t_last_done = now;
    if (st == EG_OK) {
        s->completed++;
        s->threshold_solves += q.K;
    } else {
        s->failed++;
    }
    s->latencies.push_back(ms_since(q.t_submit, now));
}

/* The control block to the launch's page, then its event. */
cudaError_t mark_end(Launch &l, cudaStream_t st)
{
    const cudaError_t e = cudaMemcpyAsync(l.lane->page, l.dctrl, sizeof(LaunchCtrl), cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaEventRecord(l.lane->ev[0], st) : e;
}

/* A query's credits, rounds and status to the host. */
eg_status fetch(eg_server *s, Query &q, int n, cudaStream_t st)
{
    const size_t nu = q.units.size();
    q.result_len = (size_t)n * q.K;
    q.result.reset(new int64_t[q.result_len]);
    const size_t bytes = sizeof(long long) * q.result_len;
    std::vector<char> tail(q.o_end - q.o_rounds); /* rounds and status lie behind one another */
    cudaError_t e;
    if (q.o_end <= kStageBlock) { /* all in one copy */
        e = copy_block_to_host(q.dF, q.o_end, s->o.device, st, [&](const char *b) {
            memcpy(q.result.get(), b, bytes);
            memcpy(tail.data(), b + q.o_rounds, tail.size());
        });
    } else {
        e = copy_to_host(q.result.get(), q.dF, bytes, s->o.device, st);
        if (e == cudaSuccess) e = copy_to_host(tail.data(), q.drounds, tail.size(), s->o.device, st);
    }
    if (e != cudaSuccess) return EG_ERR_CUDA;
    const long long *rr = (const long long *)tail.data();
    const int *ss = (const int *)(tail.data() + (q.o_status - q.o_rounds));
    eg_status r = EG_OK;
    q.rounds = 0;
    for (size_t u = 0; u < nu; u++) {
        q.rounds = std::max(q.rounds, rr[u]);
        if (r == EG_OK && ss[u] != EG_OK) r = (eg_status)ss[u];
    }
    return r;
}

/* Completion of finished micro-batches (lock held; released around the
 * copies, as around every call to the device: a submit that had to wait for
 * them took 200 us, and its query then missed the launch of the others).
 * Admitted queries and their games are erased by nobody else. */
bool reap(eg_server *s, std::unique_lock<std::mutex> &lk)
{
    bool any = false;
    for (size_t i = 0; i < s->inflight.size();) {
        Launch &l = s->inflight[i];
        cudaStream_t st = s->streams[l.stream];
        cudaError_t e = cudaEventQuery(l.lane->ev[0]);
        if (e == cudaErrorNotReady) {
            i++;
            continue;
        }
        any = true;
        const clk::time_point now = clk::now();
        std::vector<std::pair<Query *, ServedGame *>> qs;
        for (int64_t qid : l.qids) qs.push_back({s->queries[qid].get(), s->games[s->queries[qid]->game].get()});
        UnitCtrl c;
        LaunchCtrl cv;
        memset(&c, 0, sizeof c);
        const bool have = e == cudaSuccess;
        if (have) memcpy(&cv, l.lane->page, sizeof cv);
        lk.unlock();
        if (have && !l.in_tail && tail_entries(l.set, cv) > 0) {
            /* some units went to the tail: its kernels run now */
            if (launch_tail(s->launchers[(size_t)l.stream], st, l.set, l.dunits, l.tl, l.dscratch, l.dctrl, s->sms,
                            s->o.max_rounds, 0) == EG_OK &&
                mark_end(l, st) == cudaSuccess) {
                l.in_tail = true;
                i++;
                lk.lock();
                continue;
            }
            e = cudaErrorLaunchFailure;
        }
        std::vector<eg_status> status;
        for (auto &x : qs) {
            status.push_back(e == cudaSuccess ? fetch(s, *x.first, x.second->n, st) : EG_ERR_CUDA);
            free_query_device(*x.first, st);
        }
        if (e != cudaSuccess) cudaStreamSynchronize(st);
        lane_give(l.lane);
        pool_free(l.block, st);
        lk.lock();
        if (have) {
            sum_ctrl(cv, &c);
            if (!s->clock0) s->clock0 = c.t_begin;
            eg_serve_span sp;
            memset(&sp, 0, sizeof sp);
            sp.batch = l.number;
            sp.queries = (int32_t)l.qids.size();
            sp.units = l.units;
            sp.begin_ms = ((double)c.t_begin - (double)s->clock0) * 1e-6;
            sp.end_ms = ((double)c.t_end - (double)s->clock0) * 1e-6;
            s->spans.push_back(sp);
        }
        for (size_t k = 0; k < qs.size(); k++) {
            s->device_bytes -= (int64_t)qs[k].first->dbytes;
            qs[k].second->active--;
            s->admitted_now--;
            finish_query(s, *qs[k].first, status[k], now);
        }
        s->inflight.erase(s->inflight.begin() + (long)i);
    }
    if (any) s->cv_done.notify_all();
    return any;
}

/* Admission of the queries at hand, in submission order (lock held; released
 * around calls to the device). */
bool admit(eg_server *s, std::unique_lock<std::mutex> &lk)
{
    bool any = false;
    size_t left = 0;
    /* The rest of a burst is submitted meanwhile, so a few more are taken than
     * are there, but not so many that the first wait for all.  Medians of two
     * runs, bursts of 2 / 4 / 12 / 25 / 50 queries of 6 thresholds on games of
     * 1000-8000 nodes: 0.31 / 0.47 / 1.0 / 1.8 / 3.1-3.8 ms with 6; 0.31 /
     * 0.5-1.6 / 1.2-2.0 / 1.9-2.6 / 3.3-4.6 with those that are there; 0.3-0.4
     * / 0.5-0.7 / 1.2-1.8 / 1.7 / 3.4-4.2 with 16.  (Bursts of 12 took up to
     * 2.5 on other machines.) */
    size_t taken = 0;
    const size_t most = std::max<size_t>(s->pending.size(), 6);
    for (; !s->pending.empty() && taken < most && s->admitted_now < s->o.max_inflight; taken++) {
        const int64_t qid = s->pending.front();
        Query &q = *s->queries[qid];
        ServedGame &g = *s->games[q.game];
        /* routing: the grid solver for games the batched layout cannot hold,
         * and for games whose credits miss shared memory while the queue is
         * shallow (lower latency); units otherwise */
        if (g.large || (!g.fits_smem && s->pending.size() + s->ready.size() <= 2)) {
            s->pending.pop_front();
            s->large_pending.push_back(qid);
            s->cv_work.notify_all();
            any = true;
            continue;
        }
        /* plan the query's units (device pointers are filled in below) */
        q.mg.assign((size_t)q.K, 0);
        for (int k = 0; k < q.K; k++) q.mg[(size_t)k] = threshold_mg(g.hp, q.p[(size_t)k], q.d);
        std::vector<UnitDesc> units;
        std::vector<size_t> gneed;
        std::vector<long long> cost;
        int smem = 16;
        /* a large game's group: the smallest with which the queries at hand
         * leave no more units than SMs (12 queries of 6 thresholds on games of
         * 1000-8000 nodes: 2.42-2.55 -> 2.15-2.40 ms) */
        int kg = 8;
        if (g.m > kSplitEdges) {
            const long long at_hand = (long long)s->pending.size() + s->admitted_now;
            while (kg > 1 && at_hand * ((q.K + kg / 2 - 1) / (kg / 2)) <= s->sms) kg >>= 1;
        }
        eg_status ps = make_units(g.hp, PackedDev(), q.K, q.d, q.p.data(), q.mg.data(), nullptr, nullptr, nullptr,
                                  s->smem_budget, kg, &units, &gneed, &cost, &smem);
        if (ps != EG_OK) {
            s->pending.pop_front();
            finish_query(s, q, ps, clk::now());
            s->cv_done.notify_all();
            any = true;
            continue;
        }
        size_t scratch = 0;
        for (size_t x : gneed) scratch += x;
        const size_t qbytes = query_bytes(g, q.K, scratch) + units.size() * 16;
        size_t need = qbytes;
        if (!g.resident) need += packed_dev_bytes(g.hp);
        if (!make_room(s, lk, need, &left)) {
            if (s->admitted_now == 0 && s->inflight.empty()) { /* can never fit */
                s->pending.pop_front();
                finish_query(s, q, EG_ERR_OOM, clk::now());
                s->cv_done.notify_all();
                any = true;
                continue;
            }
            break; /* wait for memory to come back */
        }
        if (!g.resident) {
            void *blk = nullptr;
            const size_t pb = packed_dev_bytes(g.hp);
            eg_status st = EG_OK;
            lk.unlock();
            if (pool_alloc(&blk, pb, s->o.device, s->upload_stream) != cudaSuccess) {
                st = eg_set_error(EG_ERR_OOM, "device allocation of a game failed");
            }
            PackedDev pd;
            if (st == EG_OK) st = packed_upload(g.hp, blk, s->upload_stream, &pd);
            if (st == EG_OK && cudaStreamSynchronize(s->upload_stream) != cudaSuccess)
                st = eg_set_error(EG_ERR_CUDA, "game upload failed");
            lk.lock();
            if (st != EG_OK) {
                pool_free(blk, s->upload_stream);
                s->pending.pop_front();
                finish_query(s, q, st, clk::now());
                s->cv_done.notify_all();
                any = true;
                continue;
            }
            g.pd = pd;
            g.resident = true;
            s->uploads++;
            s->device_bytes += (int64_t)pd.bytes;
        }
        /* one device block per query: credits | thresholds | MG | rounds | status | scratch */
        const size_t nu = units.size();
        const size_t fbytes = sizeof(long long) * (size_t)g.n * q.K;
        const size_t o_thr = (fbytes + 255) & ~(size_t)255;
        const size_t o_mg = o_thr + (((size_t)q.K * sizeof(int) + 255) & ~(size_t)255);
        const size_t o_rounds = o_mg + (((size_t)q.K * sizeof(long long) + 255) & ~(size_t)255);
        const size_t o_status = o_rounds + ((nu * sizeof(long long) + 255) & ~(size_t)255);
        const size_t o_scr = o_status + ((nu * sizeof(int) + 255) & ~(size_t)255);
        const size_t total = o_scr + scratch;
        char *blk = nullptr;
        lk.unlock();
        const cudaError_t ae = pool_alloc((void **)&blk, total, s->o.device, s->upload_stream);
        if (ae != cudaSuccess) {
            /* less than there seemed to be (what the pool holds may lie in
             * pieces): without another game, later, or not at all */
            lk.lock();
            left = 0;
            if (evict_one(s)) continue;
            if (s->admitted_now > 0 || !s->inflight.empty()) break;
            s->pending.pop_front();
            finish_query(s, q, EG_ERR_OOM, clk::now());
            s->cv_done.notify_all();
            any = true;
            continue;
        }
        q.dF = (long long *)blk;
        q.dthr = (int *)(blk + o_thr);
        q.dmg = (long long *)(blk + o_mg);
        q.drounds = (long long *)(blk + o_rounds);
        q.dstatus = (int *)(blk + o_status);
        q.dscratch = scratch ? (void *)(blk + o_scr) : nullptr;
        q.dbytes = total;
        q.o_rounds = o_rounds;
        q.o_status = o_status;
        q.o_end = o_status + nu * sizeof(int);
        size_t goff = 0;
        for (size_t u = 0; u < nu; u++) {
            UnitDesc &d = units[u];
            d.E = g.pd.E;
            d.slice_off = g.pd.slice_off;
            d.orig = g.pd.orig;
            d.p = q.dthr;
            d.mg = q.dmg;
            d.F = q.dF;
            d.rounds = q.drounds + u;
            d.status = q.dstatus + u;
            if (gneed[u]) {
                d.gscratch = (char *)q.dscratch + goff;
                goff += gneed[u];
            }
        }
        q.units.swap(units);
        q.cost.swap(cost);
        q.smem = smem;
        /* thresholds and MG in one copy (through a staging buffer: no wait) */
        const CopyPart parts[2] = {{q.p.data(), 0, sizeof(int) * (size_t)q.K},
                                   {q.mg.data(), o_mg - o_thr, sizeof(long long) * (size_t)q.K}};
        cudaError_t ce = copy_parts_to_device(q.dthr, parts, 2, o_mg - o_thr + parts[1].bytes, s->o.device, s->upload_stream);
        if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&q.ready, cudaEventDisableTiming);
        if (ce == cudaSuccess) ce = cudaEventRecord(q.ready, s->upload_stream);
        lk.lock();
        if (ce != cudaSuccess) {
            cudaGetLastError();
            free_query_device(q, s->upload_stream);
            s->pending.pop_front();
            finish_query(s, q, EG_ERR_CUDA, clk::now());
            s->cv_done.notify_all();
            any = true;
            continue;
        }
        s->device_bytes += (int64_t)q.dbytes;
        g.active++;
        g.last_use = ++s->tick;
        q.state = EG_QUERY_RUNNING;
        s->admitted++;
        s->admitted_now++;
        s->pending.pop_front();
        s->ready.push_back(qid);
        any = true;
    }
    return any;
}

/* Device side of one micro-batch of the queries l.qids, up to its launch
 * (lock not held). */
eg_status prepare_batch(eg_server *s, Launch &l, const std::vector<Query *> &qs)
{
    std::vector<UnitDesc> all;
    std::vector<long long> cost;
    for (Query *q : qs) {
        all.insert(all.end(), q->units.begin(), q->units.end());
        cost.insert(cost.end(), q->cost.begin(), q->cost.end());
    }
    UnitSet &S = l.set;
    group_units(all, cost, std::vector<size_t>(all.size(), 0), &S, nullptr);
    l.stream = s->next_stream;
    l.units = (int)S.units.size();
    s->next_stream = (s->next_stream + 1) % s->o.streams;
    cudaStream_t st = s->streams[l.stream];
    for (Query *q : qs) cudaStreamWaitEvent(st, q->ready, 0);
    const size_t tsb = tail_scratch_bytes(S, s->sms);
    const size_t ub = (sizeof(UnitDesc) * S.units.size() + 255) & ~(size_t)255;
    const size_t cb = (sizeof(LaunchCtrl) + 255) & ~(size_t)255, tb = (tail_bytes(S) + 255) & ~(size_t)255;
    cudaError_t e = pool_alloc(&l.block, ub + cb + tb + tsb, s->o.device, st);
    if (e != cudaSuccess) return EG_ERR_OOM;
    char *at = (char *)l.block;
    l.dunits = (UnitDesc *)at;
    l.dctrl = (LaunchCtrl *)(at + ub);
    if (tsb) l.dscratch = at + ub + cb + tb;
    e = copy_to_device(l.dunits, S.units.data(), sizeof(UnitDesc) * S.units.size(), s->o.device, st);
    if (e != cudaSuccess) return EG_ERR_CUDA;
    l.lane = lane_take(s->o.device);
    if (!l.lane) return EG_ERR_CUDA;
    return tail_upload(S, at + ub + cb, st, &l.tl);
}

/* Launches a prepared micro-batch (lock not held). */
eg_status start_batch(eg_server *s, Launch &l)
{
    cudaStream_t st = s->streams[l.stream];
    int grid = 0;
    eg_status ls = launch_units(s->launchers[(size_t)l.stream], st, l.set, l.dunits, l.tl, l.dctrl, s->o.block, s->sms,
                                s->o.max_rounds, 0, &grid);
    if (ls == EG_OK && mark_end(l, st) != cudaSuccess) ls = EG_ERR_CUDA;
    if (ls != EG_OK) cudaStreamSynchronize(st); /* nothing may write the lane's page any more */
    return ls;
}

/* A micro-batch under way, or the end of its queries (lock held). */
void account_batch(eg_server *s, Launch &l, eg_status ls)
{
    if (ls == EG_OK) {
        l.number = s->micro_batches++;
        s->inflight.push_back(std::move(l));
        return;
    }
    cudaStream_t st = s->streams[l.stream];
    cudaGetLastError();
    const clk::time_point now = clk::now();
    for (int64_t qid : l.qids) {
        Query &q = *s->queries[qid];
        s->device_bytes -= (int64_t)q.dbytes;
        free_query_device(q, st);
        s->games[q.game]->active--;
        s->admitted_now--;
        finish_query(s, q, ls, now);
    }
    lane_give(l.lane);
    pool_free(l.block, st);
    s->cv_done.notify_all();
}

/* Launches the admitted queries (lock held, but not during it): in two micro-batches where two
 * streams are free, the queries dealt heaviest first, so that the first's
 * read-back overlaps the second's run.  Both are prepared before the first
 * is launched: they start a kernel launch apart. */
bool launch_ready(eg_server *s, std::unique_lock<std::mutex> &lk)
{
    const int free_streams = s->o.streams - (int)s->inflight.size();
    if (s->ready.empty() || free_streams <= 0) return false;
    std::vector<int64_t> ready;
    ready.swap(s->ready);
    auto cost_of = [&](int64_t qid) {
        long long c = 0;
        for (long long x : s->queries[qid]->cost) c += x;
        return c;
    };
    std::stable_sort(ready.begin(), ready.end(), [&](int64_t a, int64_t b) { return cost_of(a) > cost_of(b); });
    const size_t parts = std::min<size_t>({2, (size_t)free_streams, ready.size()});
    std::vector<Launch> ls(parts);
    std::vector<eg_status> done(parts, EG_OK);
    std::vector<std::vector<Query *>> qs(parts);
    for (size_t i = 0; i < ready.size(); i++) {
        ls[i % parts].qids.push_back(ready[i]);
        qs[i % parts].push_back(s->queries[ready[i]].get());
    }
    lk.unlock();
    for (size_t k = 0; k < parts; k++) done[k] = prepare_batch(s, ls[k], qs[k]);
    for (size_t k = 0; k < parts; k++)
        if (done[k] == EG_OK) done[k] = start_batch(s, ls[k]);
    lk.lock();
    for (size_t k = 0; k < parts; k++) account_batch(s, ls[k], done[k]);
    return true;
}

void worker_main(eg_server *s)
{
    constexpr int kSpins = 2000;
    int quiet = 0;
    cudaSetDevice(s->o.device);
    std::unique_lock<std::mutex> lk(s->mu);
    for (;;) {
        bool progress = reap(s, lk);
        progress |= admit(s, lk);
        progress |= launch_ready(s, lk);
        if (s->stop && s->pending.empty() && s->ready.empty() && s->inflight.empty()) break;
        if (progress) {
            quiet = 0;
        } else if (!s->inflight.empty() && ++quiet < kSpins) {
            /* a micro-batch of certified units ends within a millisecond:
             * look again at once instead of sleeping through its end */
            lk.unlock();
            std::this_thread::yield();
            lk.lock();
        } else {
            s->cv_work.wait_for(lk, std::chrono::microseconds(200));
        }
    }
}

/* Large games: one threshold at a time on the capped persistent grid. */
void large_main(eg_server *s)
{
    cudaSetDevice(s->o.device);
    std::unique_lock<std::mutex> lk(s->mu);
    for (;;) {
        if (s->large_pending.empty()) {
            if (s->stop) break;
            s->cv_work.wait_for(lk, std::chrono::milliseconds(2));
            continue;
        }
        const int64_t qid = s->large_pending.front();
        s->large_pending.pop_front();
        Query &q = *s->queries[qid];
        ServedGame &g = *s->games[q.game];
        g.active++;
        q.state = EG_QUERY_RUNNING;
        s->admitted++;
        eg_game base = g.view();
        const int K = q.K, d = q.d;
        const std::vector<int> p = q.p;
        lk.unlock();
        std::unique_ptr<int64_t[]> result(new int64_t[(size_t)g.n * K]());
        std::vector<int32_t> wt((size_t)g.m);
        eg_status st = EG_OK;
        long long rounds = 0;
        for (int k = 0; k < K && st == EG_OK; k++) {
            for (long long j = 0; j < g.m; j++) {
                const long long x = (long long)base.weight[j] * d - p[(size_t)k];
                if (x < INT32_MIN || x > INT32_MAX) {
                    st = eg_set_error(EG_ERR_OVERFLOW, "shifted weight out of int32 range");
                    break;
                }
                wt[(size_t)j] = (int32_t)x;
            }
            if (st != EG_OK) break;
            eg_game tg = base;
            tg.weight = wt.data();
            eg_opts o;
            eg_opts_default(&o);
            o.device = s->o.device;
            o.credit_bits = 64;
            o.max_rounds = s->o.max_rounds;
            o.grid_ctas = s->o.large_ctas;
            eg_dgame *dg = nullptr;
            st = eg_dgame_upload(&tg, &o, &dg);
            eg_stats ss;
            if (st == EG_OK) st = eg_dgame_solve(dg, &o, &ss);
            if (st == EG_OK) st = eg_dgame_credits_i64(dg, result.get() + (size_t)k * g.n);
            if (st == EG_OK) rounds = std::max(rounds, (long long)ss.rounds);
            eg_dgame_free(dg);
        }
        lk.lock();
        q.result.swap(result);
        q.result_len = (size_t)g.n * K;
        q.rounds = rounds;
        g.active--;
        finish_query(s, q, st, clk::now());
        s->cv_done.notify_all();
    }
}

}  // namespace

extern "C" eg_status eg_serve_create(const eg_serve_opts *opts, eg_server **out)
{
    if (!out) return eg_set_error(EG_ERR_INVALID, "out is NULL");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return eg_set_error(EG_ERR_NO_DEVICE, "no CUDA device available");
    }
    eg_server *s = new eg_server();
    memset(&s->o, 0, sizeof s->o);
    if (opts) s->o = *opts;
    if (s->o.device < 0 || s->o.device >= count) {
        delete s;
        return eg_set_error(EG_ERR_INVALID, "device %d not available", opts ? opts->device : 0);
    }
    if (s->o.max_inflight <= 0) s->o.max_inflight = 1024;
    if (s->o.streams <= 0) s->o.streams = 4;
    if (s->o.block <= 0) s->o.block = 1024;
    if (s->o.hbm_reserve_bytes <= 0) s->o.hbm_reserve_bytes = 1ll << 30;
    if (s->o.max_rounds == 0) s->o.max_rounds = -1;
    cudaSetDevice(s->o.device);
    cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, s->o.device);
    if (s->o.large_ctas <= 0) s->o.large_ctas = std::max(1, s->sms - s->sms / 4);
    {
        eg_status ks = unit_kernel_setup(s->o.device);
        if (ks != EG_OK) {
            delete s;
            return ks;
        }
        s->smem_budget = unit_smem_budget(s->o.device);
    }
    for (int i = 0; i < s->o.streams; i++) {
        cudaStream_t st;
        if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
            for (cudaStream_t x : s->streams) cudaStreamDestroy(x);
            delete s;
            return eg_set_error(EG_ERR_CUDA, "stream creation failed");
        }
        s->streams.push_back(st);
        s->launchers.emplace_back();
        if (s->launchers.back().init() != EG_OK) {
            for (UnitLauncher &L : s->launchers) L.destroy();
            for (cudaStream_t x : s->streams) cudaStreamDestroy(x);
            delete s;
            return eg_set_error(EG_ERR_CUDA, "stream creation failed");
        }
    }
    if (cudaStreamCreateWithFlags(&s->upload_stream, cudaStreamNonBlocking) != cudaSuccess) {
        for (UnitLauncher &L : s->launchers) L.destroy();
        for (cudaStream_t x : s->streams) cudaStreamDestroy(x);
        delete s;
        return eg_set_error(EG_ERR_CUDA, "stream creation failed");
    }
    s->t0 = s->t_last_done = clk::now();
    s->worker = std::thread(worker_main, s);
    s->large_worker = std::thread(large_main, s);
    *out = s;
    return EG_OK;
}

extern "C" eg_status eg_serve_add_game(eg_server *s, const eg_game *game, int64_t *game_id)
{
    if (!s || !game || !game_id) return eg_set_error(EG_ERR_INVALID, "NULL argument");
    eg_status v = eg_validate(game);
    if (v != EG_OK) return v;
    auto g = std::make_unique<ServedGame>();
    g->n = game->num_nodes;
    g->n0 = game->num_nodes0;
    g->m = game->num_edges;
    g->rp.assign(game->row_ptr, game->row_ptr + game->num_nodes + 1);
    g->succ.assign(game->succ, game->succ + game->num_edges);
    g->w.assign(game->weight, game->weight + game->num_edges);
    if (game->owner) {
        g->own.assign(game->owner, game->owner + game->num_nodes);
        g->has_owner = true;
    }
    g->large = game->num_nodes > kBatchMaxGameNodes;
    if (!g->large) {
        /* the packed layout the unit kernel reads (host image, uploaded on admission) */
        eg_status ps = pack_game(*game, &g->hp);
        if (ps != EG_OK) return ps;
        g->fits_smem = (long long)g->hp.rows() * 4 <= (long long)s->smem_budget;
    }
    std::lock_guard<std::mutex> lk(s->mu);
    g->id = s->next_game++;
    *game_id = g->id;
    s->games[g->id] = std::move(g);
    return EG_OK;
}

extern "C" eg_status eg_serve_remove_game(eg_server *s, int64_t game_id)
{
    if (!s) return eg_set_error(EG_ERR_INVALID, "server is NULL");
    std::unique_lock<std::mutex> lk(s->mu);
    auto it = s->games.find(game_id);
    if (it == s->games.end()) return eg_set_error(EG_ERR_NOT_FOUND, "no game %lld", (long long)game_id);
    for (auto &kv : s->queries)
        if (kv.second->game == game_id && kv.second->state <= EG_QUERY_RUNNING)
            return eg_set_error(EG_ERR_BUSY, "game %lld still has queries in flight", (long long)game_id);
    if (it->second->resident) drop_resident(s, *it->second);
    s->games.erase(it);
    return EG_OK;
}

extern "C" eg_status eg_serve_submit(eg_server *s, int64_t game_id, const int32_t *p, int32_t K, int32_t d,
                                     int64_t *query_id)
{
    if (!s || !p || !query_id) return eg_set_error(EG_ERR_INVALID, "NULL argument");
    if (K < 1 || K > EG_BATCH_MAX_K) return eg_set_error(EG_ERR_INVALID, "K must be in [1, %d]", EG_BATCH_MAX_K);
    if (d < 1) return eg_set_error(EG_ERR_INVALID, "scale d must be >= 1");
    std::lock_guard<std::mutex> lk(s->mu);
    if (s->stop) return eg_set_error(EG_ERR_BUSY, "server is shutting down");
    if (!s->games.count(game_id)) return eg_set_error(EG_ERR_NOT_FOUND, "no game %lld", (long long)game_id);
    auto q = std::make_unique<Query>();
    q->id = s->next_query++;
    q->game = game_id;
    q->K = K;
    q->d = d;
    q->p.assign(p, p + K);
    q->t_submit = clk::now();
    *query_id = q->id;
    s->pending.push_back(q->id);
    s->queries[q->id] = std::move(q);
    s->submitted++;
    s->cv_work.notify_all();
    return EG_OK;
}

extern "C" eg_status eg_serve_poll(eg_server *s, int64_t query_id, int32_t *state, double *latency_ms)
{
    if (!s) return eg_set_error(EG_ERR_INVALID, "server is NULL");
    std::lock_guard<std::mutex> lk(s->mu);
    auto it = s->queries.find(query_id);
    if (it == s->queries.end()) return eg_set_error(EG_ERR_NOT_FOUND, "no query %lld", (long long)query_id);
    const Query &q = *it->second;
    if (state) *state = q.state;
    if (latency_ms) *latency_ms = q.state >= EG_QUERY_DONE ? ms_since(q.t_submit, q.t_done) : ms_since(q.t_submit, clk::now());
    return EG_OK;
}

extern "C" eg_status eg_serve_wait(eg_server *s, int64_t query_id, double timeout_ms)
{
    if (!s) return eg_set_error(EG_ERR_INVALID, "server is NULL");
    std::unique_lock<std::mutex> lk(s->mu);
    const clk::time_point until = clk::now() + std::chrono::microseconds((long long)(timeout_ms * 1000));
    for (;;) {
        auto it = s->queries.find(query_id);
        if (it == s->queries.end()) return eg_set_error(EG_ERR_NOT_FOUND, "no query %lld", (long long)query_id);
        if (it->second->state >= EG_QUERY_DONE) return EG_OK;
        if (timeout_ms >= 0 && clk::now() >= until) return eg_set_error(EG_ERR_TIMEOUT, "query %lld not finished", (long long)query_id);
        s->cv_done.wait_for(lk, std::chrono::milliseconds(5));
    }
}

extern "C" eg_status eg_serve_result(eg_server *s, int64_t query_id, int64_t *credits, int64_t *rounds)
{
    if (!s || !credits) return eg_set_error(EG_ERR_INVALID, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    auto it = s->queries.find(query_id);
    if (it == s->queries.end()) return eg_set_error(EG_ERR_NOT_FOUND, "no query %lld", (long long)query_id);
    Query &q = *it->second;
    if (q.state == EG_QUERY_FAILED) {
        const eg_status st = q.status;
        s->queries.erase(it);
        return eg_set_error(st, "query %lld failed with status %d", (long long)query_id, (int)st);
    }
    if (q.state != EG_QUERY_DONE) return eg_set_error(EG_ERR_BUSY, "query %lld not finished", (long long)query_id);
    memcpy(credits, q.result.get(), sizeof(int64_t) * q.result_len);
    if (rounds) *rounds = q.rounds;
    s->queries.erase(it);
    return EG_OK;
}

extern "C" eg_status eg_serve_stats_get(eg_server *s, eg_serve_stats *out)
{
    if (!s || !out) return eg_set_error(EG_ERR_INVALID, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    memset(out, 0, sizeof *out);
    out->submitted = s->submitted;
    out->admitted = s->admitted;
    out->completed = s->completed;
    out->failed = s->failed;
    out->games_registered = (int64_t)s->games.size();
    for (auto &kv : s->games) out->games_resident += kv.second->resident;
    out->game_uploads = s->uploads;
    out->evictions = s->evictions;
    out->micro_batches = s->micro_batches;
    out->threshold_solves = s->threshold_solves;
    std::vector<double> lat = s->latencies;
    if (!lat.empty()) {
        std::sort(lat.begin(), lat.end());
        auto pct = [&](double q) { return lat[std::min(lat.size() - 1, (size_t)(q * (double)(lat.size() - 1) + 0.5))]; };
        out->latency_p50_ms = pct(0.50);
        out->latency_p99_ms = pct(0.99);
        out->latency_max_ms = lat.back();
        double sum = 0;
        for (double x : lat) sum += x;
        out->latency_mean_ms = sum / (double)lat.size();
    }
    out->elapsed_s = std::chrono::duration<double>(s->t_last_done - s->t0).count();
    if (out->elapsed_s > 0) {
        out->queries_per_s = (double)s->completed / out->elapsed_s;
        out->solves_per_s = (double)s->threshold_solves / out->elapsed_s;
    }
    out->device_bytes = s->device_bytes;
    return EG_OK;
}

extern "C" eg_status eg_serve_trace(eg_server *s, eg_serve_span *spans, int32_t cap, int32_t *count)
{
    if (!s || !count || (cap > 0 && !spans)) return eg_set_error(EG_ERR_INVALID, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    const int32_t n = (int32_t)s->spans.size();
    for (int32_t i = 0; i < n && i < cap; i++) spans[i] = s->spans[(size_t)i];
    *count = n;
    return EG_OK;
}

extern "C" eg_status eg_serve_destroy(eg_server *s)
{
    if (!s) return EG_OK;
    {
        std::lock_guard<std::mutex> lk(s->mu);
        s->stop = true;
        s->cv_work.notify_all();
    }
    s->worker.join();
    s->large_worker.join();
    cudaSetDevice(s->o.device);
    for (auto &kv : s->queries) free_query_device(*kv.second, s->upload_stream);
    for (auto &kv : s->games)
        if (kv.second->resident) pool_free(kv.second->pd.block, s->upload_stream);
    cudaStreamSynchronize(s->upload_stream);
    for (UnitLauncher &L : s->launchers) L.destroy();
    for (cudaStream_t st : s->streams) cudaStreamDestroy(st);
    cudaStreamDestroy(s->upload_stream);
    delete s;
    return EG_OK;
}
