"""GPU tests of the serving loop: results in the mix equal results alone,
admission by free device memory, the large-game path, statistics."""
from __future__ import annotations

import time

import numpy as np
import pytest

import egsolver_b200 as eg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def mixed_games(num=16, seed=13):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(num):
        n = int(np.exp(rng.uniform(np.log(60), np.log(3000))))
        out.append(eg.generate(5, n, min(60, n - 1), int(rng.integers(5, 40)), 500 + i, param=6))
    return out


def alone(game, p, d):
    """The same query solved alone, outside the server (batched kernel, one game)."""
    with eg.Batch([game], thresholds=len(p), scale=d) as b:
        b.set_thresholds(np.asarray(p, np.int32).reshape(1, -1))
        b.solve()
        return b.credits(0)


def test_results_in_the_mix_equal_results_alone():
    games = mixed_games()
    rng = np.random.default_rng(1)
    d = 8
    with eg.Server(streams=3) as srv:
        gids = [srv.add_game(g) for g in games]
        queries = []
        for rep in range(3):  # several queries per game: the game stays resident
            for gi, gid in enumerate(gids):
                K = int(rng.integers(1, 9))
                W = int(np.abs(games[gi].weight).max())
                p = rng.integers(-8 * W, 8 * W + 1, size=K).astype(np.int32)
                queries.append((srv.submit(gid, p, d), gi, p))
        for qid, gi, p in queries:
            srv.wait(qid, 120_000)
        checked = 0
        for qid, gi, p in queries:
            got, _ = srv.result(qid)
            np.testing.assert_array_equal(got, alone(games[gi], p, d))
            if checked < 6:  # and against the oracle, not only the GPU alone
                for k in range(len(p)):
                    want, _ = O.eg_solve(eg.threshold_game(games[gi], int(p[k]), d), bits=64)
                    np.testing.assert_array_equal(got[k], want)
                checked += 1
        st = srv.stats()
        assert st["completed"] == len(queries) and st["failed"] == 0
        assert st["game_uploads"] == len(games)  # uploaded once, reused across queries
        assert st["latency_p99_ms"] >= st["latency_p50_ms"] > 0
        assert st["micro_batches"] >= 1


def test_served_results_match_the_oracle():
    games = mixed_games(4, seed=3)
    with eg.Server() as srv:
        for g in games:
            gid = srv.add_game(g)
            p = np.array([-40, 0, 25], dtype=np.int32)
            qid = srv.submit(gid, p, 4)
            srv.wait(qid, 60_000)
            got, _ = srv.result(qid)
            for k in range(3):
                want, _ = O.eg_solve(eg.threshold_game(g, int(p[k]), 4), bits=64)
                np.testing.assert_array_equal(got[k], want)


def test_large_game_runs_on_the_grid_path():
    n = (1 << 19) + 4096
    g = eg.generate(1, n, 3, 4, 99)
    p = np.array([-3, 1], dtype=np.int32)
    with eg.Server(large_ctas=74) as srv:
        gid = srv.add_game(g)
        small = mixed_games(3, seed=8)
        sids = [srv.add_game(x) for x in small]
        qid = srv.submit(gid, p, 2)
        others = [srv.submit(s, np.array([0, 3], np.int32), 2) for s in sids]
        srv.wait(qid, 300_000)
        got, _ = srv.result(qid)
        for k in range(2):
            # the oracle's worklist needs far too long on this game: its
            # fixed-point check instead (a fixed point reached by lifting
            # from 0 is the least one)
            assert O.count_inconsistent(eg.threshold_game(g, int(p[k]), 2), got[k]) == 0
        for s, q in zip(small, others):
            srv.wait(q, 60_000)
            r, _ = srv.result(q)
            for k, pk in enumerate((0, 3)):
                want, _ = O.eg_solve(eg.threshold_game(s, pk, 2), bits=64)
                np.testing.assert_array_equal(r[k], want)


def test_wide_weight_requests_match_the_oracle():
    """Requests shaped like the served workload's: weights up to 10^4 and
    thresholds up to 8W, so credits need 64 bits; games of a few thousand
    vertices (the oracle finishes them)."""
    from egsolver_b200 import workloads

    reqs = [r for r in workloads.cfg5_requests(40, n_max=6000) if r[0].num_nodes <= 6000]
    reqs = sorted(reqs, key=lambda r: -int(np.abs(r[0].weight).max()))[:4]
    assert int(np.abs(reqs[0][0].weight).max()) > 1000
    with eg.Server() as srv:
        qs = []
        for g, p, d in reqs:
            qs.append((srv.submit(srv.add_game(g), p[:6], d), g, p[:6], d))
        for qid, g, p, d in qs:
            srv.wait(qid, 300_000)
            got, _ = srv.result(qid)
            for k in range(len(p)):
                want, st = O.eg_solve(eg.threshold_game(g, int(p[k]), d), bits=64)
                np.testing.assert_array_equal(got[k], want)


def test_micro_batches_overlap_on_the_device():
    """A query submitted while an earlier micro-batch still runs starts on
    the SMs that batch leaves free: the device-clock spans of the two
    micro-batches intersect."""
    games = mixed_games(6, seed=21)
    d = 8
    with eg.Server(streams=4) as srv:
        gids = [srv.add_game(g) for g in games]
        # a long first micro-batch: thresholds that drive every credit to TOP
        W = [int(np.abs(g.weight).max()) for g in games]
        q1 = [srv.submit(gids[i], np.array([7 * W[i] * d // 8 + 1] * 4, np.int32), d) for i in range(3)]
        import time

        time.sleep(0.05)
        q2 = [srv.submit(gids[i], np.array([0, 1], np.int32), d) for i in range(3, 6)]
        for q in q1 + q2:
            srv.wait(q, 300_000)
        spans = srv.trace()
        assert len(spans) >= 2
        first = spans[0]
        later = [s for s in spans[1:]]
        assert any(s["begin_ms"] < first["end_ms"] for s in later), spans


def test_admission_refuses_what_can_never_fit():
    g = mixed_games(1)[0]
    with eg.Server(hbm_reserve_bytes=1 << 60) as srv:  # nothing may be used
        gid = srv.add_game(g)
        qid = srv.submit(gid, np.array([0], np.int32), 1)
        srv.wait(qid, 30_000)
        state, _ = srv.poll(qid)
        assert state == 3  # EG_QUERY_FAILED
        with pytest.raises(eg.EGError) as ei:
            srv.result(qid)
        assert ei.value.name == "EG_ERR_OOM"


def test_unknown_game_and_bad_arguments():
    with eg.Server() as srv:
        with pytest.raises(eg.EGError) as ei:
            srv.submit(12345, [0])
        assert ei.value.name == "EG_ERR_NOT_FOUND"
        gid = srv.add_game(mixed_games(1)[0])
        with pytest.raises(eg.EGError):
            srv.submit(gid, np.zeros(40, np.int32))  # K > 32


@pytest.mark.parametrize("n", [8176, 8180, 9000])
def test_results_at_the_edge_of_one_copy(n):
    """A query's block of credits, thresholds, rounds and status: just within
    the 512 KB that one copy reads, and just past them."""
    g = eg.generate(1, n, 4, 20, n)
    p = np.array([-90, -40, -9, -3, 0, 5, 33, 88], np.int32)
    with eg.Server() as srv:
        gid = srv.add_game(g)
        qids = [srv.submit(gid, p + i, 4) for i in range(3)]
        for i, q in enumerate(qids):
            srv.wait(q, 120_000)
            got, _ = srv.result(q)
            np.testing.assert_array_equal(got, alone(g, p + i, 4))


def test_threads_submit_while_queries_run():
    import threading

    games = mixed_games(6, seed=3)
    want = {}
    for i, g in enumerate(games):
        for r in range(4):
            p = np.array([-9 + r, 0, 7 * r], np.int32)
            want[i, r] = (p, alone(g, p, 8))
    errors = []
    with eg.Server(streams=3) as srv:
        gids = [srv.add_game(g) for g in games]

        def client(r):
            try:
                for _ in range(3):
                    qids = [srv.submit(gids[i], want[i, r][0], 8) for i in range(len(games))]
                    extra = srv.add_game(games[r])
                    srv.wait(srv.submit(extra, want[r, r][0], 8), 120_000)
                    for i, q in enumerate(qids):
                        srv.wait(q, 120_000)
                        np.testing.assert_array_equal(srv.result(q)[0], want[i, r][1])
            except Exception as e:  # reported by the main thread
                errors.append(e)

        ts = [threading.Thread(target=client, args=(r,)) for r in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not errors, errors
        assert srv.stats()["completed"] == 4 * 3 * 7


def test_evicted_games_make_room():
    """Four games of about 30 MB each where the reserve leaves 40 MB, and what
    the pool keeps comes to 64 MB at most: every query is admitted, after
    evictions, one game at a time."""
    torch = pytest.importorskip("torch")
    games = [eg.generate(1, 30000, 250, 20, 70 + i) for i in range(4)]
    with eg.Server() as s:  # modules and streams before the look at the free memory
        gid = s.add_game(games[0])
        s.wait(s.submit(gid, [900]))
    with eg.Server(hbm_reserve_bytes=torch.cuda.mem_get_info()[0] - (40 << 20)) as s:
        gids = [s.add_game(g) for g in games]
        for turn in range(2):
            for i, gid in enumerate(gids):
                q = s.submit(gid, [900])  # above every weight: all TOP, at once
                s.wait(q)
                assert np.all(s.result(q)[0] == eg.EG_TOP64)
        st = s.stats()
        assert st["failed"] == 0 and 4 <= st["evictions"] <= 7


def test_small_queries_run_beside_the_grid_solver():
    """A path of 600,000 vertices keeps the grid solver busy for about a
    second; a query of a small game that comes meanwhile does not wait for it."""
    n = 600_000
    weight = np.full(n, -1)
    weight[-1] = 0
    deep = eg.Game(row_ptr=np.arange(n + 1), succ=np.minimum(np.arange(1, n + 1), n - 1), weight=weight, num_nodes0=n // 2)
    small = eg.generate(4, 2000, 16, 100, 3, param=2)
    with eg.Server() as s:
        a, b = s.add_game(deep), s.add_game(small)
        s.wait(s.submit(b, [0, 10]))
        q = s.submit(a, [0])
        time.sleep(0.1)
        q2 = s.submit(b, [0, 10])
        s.wait(q2)
        time.sleep(0.1)  # past the end of a solve that the small query waited for
        assert s.poll(q)[0] == 1  # still running
        s.wait(q)
        np.testing.assert_array_equal(s.result(q)[0][0], np.arange(n)[::-1])
