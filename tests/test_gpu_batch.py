"""GPU parity of the batched solver: every (game, threshold) of a batch equals
the oracle's solve of the energy game with weights w*d - p."""
from __future__ import annotations

import numpy as np
import pytest

import egsolver_b200 as eg
from egsolver_b200 import workloads
from oracle import oracle as O
from tests.test_gpu_sweep import strip, want

pytestmark = pytest.mark.gpu


def small_batch(num=18, seed=5):
    rng = np.random.default_rng(seed)
    games = []
    for i in range(num):
        n = int(rng.integers(40, 1500))
        kind = [1, 2, 4, 5][i % 4]
        deg = {1: 3, 2: min(n - 1, 64), 4: 16, 5: 30}[kind]
        games.append(eg.generate(kind, n, deg, int(rng.integers(3, 60)), 77 + i, param=2 if kind == 4 else 6))
    return games


def check_batch(b, games, p, d):
    for g, game in enumerate(games):
        got = b.credits(g)
        for k in range(p.shape[1]):
            want, st = O.eg_solve(eg.threshold_game(game, int(p[g, k]), d), bits=64)
            assert st["finished"]
            np.testing.assert_array_equal(got[k], want, err_msg=f"game {g} threshold {k} (p={p[g, k]})")


@pytest.mark.parametrize("K", [1, 3, 8, 32])
def test_small_batch_all_thresholds(K):
    games = small_batch()
    rng = np.random.default_rng(K)
    d = 4
    p = rng.integers(-60, 61, size=(len(games), K)).astype(np.int32)
    with eg.Batch(games, thresholds=K, scale=d) as b:
        b.set_thresholds(p)
        _, st = b.solve()
        assert st.games_failed == 0 and st.num_games == len(games)
        check_batch(b, games, p, d)


def test_cfg4_games_subset():
    games = [g for g in workloads.cfg4_games(64) if g.num_nodes <= 2600][:6]
    p_all, d = workloads.cfg4_thresholds(64)
    p = p_all[: len(games)]
    with eg.Batch(games, thresholds=8, scale=d) as b:
        b.set_thresholds(p)
        _, st = b.solve()
        assert st.edges > 0
        check_batch(b, games, p, d)


def test_graph_replay_with_new_thresholds():
    games = small_batch(10, seed=9)
    d = 2
    with eg.Batch(games, thresholds=4, scale=d, use_graph=True) as b:
        for rep in range(3):
            p = np.random.default_rng(rep).integers(-30, 31, size=(len(games), 4)).astype(np.int32)
            b.set_thresholds(p)
            _, st = b.solve()
            assert st.graph_replayed == (1 if rep > 0 else 0)
            check_batch(b, games, p, d)


def test_autotuner_then_solve():
    games = small_batch(12, seed=2)
    p = np.random.default_rng(1).integers(-40, 41, size=(len(games), 8)).astype(np.int32)
    with eg.Batch(games, thresholds=8, scale=3) as b:
        b.set_thresholds(p)
        blk = b.tune()
        assert blk in (512, 1024)
        _, st = b.solve()
        assert st.block == blk
        assert st.num_units == len(games)     # K = 8: the group size stays at eight
        check_batch(b, games, p, 3)


def test_unit_variants_match_the_oracle():
    """Every kind of work unit: 32- and 64-bit credits, 4- and 8-byte slots,
    groups of 8/4/2/1 thresholds (K = 15 splits into 8 + 4 + 2 + 1), and
    hybrid credits (shared memory plus global scratch) for a game too large
    for one CTA's shared memory."""
    rng = np.random.default_rng(21)
    games = [
        eg.generate(4, 900, 9, 60, 301, param=2),        # narrow slots, 32-bit credits
        eg.generate(4, 700, 6, 20000, 302, param=2),     # |w| > 32766 -> 8-byte slots
        eg.generate(1, 600, 3, 3, 303),                  # tiny weights, big thresholds -> 64-bit credits
        eg.generate(4, 66000, 3, 5, 304, param=2),       # > 65534 rows: 8-byte slots; hybrid credits
    ]
    d = 3
    K = 15
    p = np.zeros((len(games), K), dtype=np.int32)
    p[0] = rng.integers(-150, 151, K)
    p[1] = rng.integers(-40000, 40001, K)
    p[2] = rng.integers(-(1 << 29), 1 << 29, K)         # MG far above 2^30 for positive p
    p[3] = rng.integers(-14, -2, K)                     # short climbs: the test stays quick
    with eg.Batch(games, thresholds=K, scale=d) as b:
        b.set_thresholds(p)
        _, st = b.solve()
        assert st.games_failed == 0
        # 8+4+2+1 groups per small game; the large one (credits beyond one
        # CTA's shared memory) as 15 hybrid units of one threshold
        assert st.num_units == 3 * 4 + 15
        for g, game in enumerate(games):
            got = b.credits(g)
            for k in range(K):
                tg = eg.threshold_game(game, int(p[g, k]), d)
                if game.num_nodes > 10_000:
                    assert O.count_inconsistent(tg, got[k]) == 0, f"game {g} threshold {k}"
                else:
                    want, _ = O.eg_solve(tg, bits=64)
                    np.testing.assert_array_equal(got[k], want, err_msg=f"game {g} threshold {k}")


@pytest.mark.parametrize("group_max", [1, 2, 4, 8])
def test_group_sizes_give_identical_credits(group_max):
    games = small_batch(8, seed=31)
    p = np.random.default_rng(4).integers(-50, 51, size=(len(games), 8)).astype(np.int32)
    with eg.Batch(games, thresholds=8, scale=2, group_max=group_max) as b:
        b.set_thresholds(p)
        b.solve()
        check_batch(b, games, p, 2)


def test_round_cap_marks_games():
    games = [workloads.cfg1()]
    p = np.array([[40]], dtype=np.int32)  # strongly negative weights: long climb to TOP
    with eg.Batch(games, thresholds=1, scale=1, max_rounds=2) as b:
        b.set_thresholds(p)
        status, st = b.solve(raise_on_error=False)
        assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_LOOPCAP"
        rounds, gst = b.game_result(0)
        assert rounds == 2 and eg._ffi.STATUS_NAMES[gst] == "EG_ERR_LOOPCAP"


def test_owner_arrays_in_a_batch():
    g = workloads.cfg1(300)
    own = g.owners().copy()
    h = eg.Game(row_ptr=g.row_ptr, succ=g.succ, weight=g.weight, owner=own)
    p = np.array([[0, 5], [0, 5]], dtype=np.int32)
    with eg.Batch([g, h], thresholds=2, scale=1) as b:
        b.set_thresholds(p)
        b.solve()
        np.testing.assert_array_equal(b.credits(0), b.credits(1))
        check_batch(b, [g], p[:1], 1)  # the oracle takes the split convention of g


def test_cfg4_game_near_the_top_of_the_size_range():
    """A cfg4 game of 17,931 vertices at all 8 thresholds (one of them
    drives every credit to TOP, which runs into the cluster tail): two
    thresholds against the oracle's worklist solve, all eight by the
    oracle's fixed-point check."""
    games = workloads.cfg4_games(64)
    p_all, d = workloads.cfg4_thresholds(64)
    g = games[34]
    assert g.num_nodes == 17931
    with eg.Batch([g], thresholds=8, scale=d) as b:
        b.set_thresholds(p_all[34:35])
        _, st = b.solve()
        assert st.games_failed == 0
        got = b.credits(0)
    for k in range(8):
        tg = eg.threshold_game(g, int(p_all[34, k]), d)
        assert O.count_inconsistent(tg, got[k]) == 0, f"threshold {k}"
    for k in (0, 2):
        want, _ = O.eg_solve(eg.threshold_game(g, int(p_all[34, k]), d), bits=64)
        np.testing.assert_array_equal(got[k], want)


@pytest.mark.parametrize("tail_sweeps,tail_cluster", [(1, 16), (4, 8), (2, 2)])
def test_tail_shapes_give_identical_credits(tail_sweeps, tail_cluster):
    """Every (game, threshold) straight to the cluster tail, at several
    sweeps per cluster barrier and cluster sizes (CTAs past the rows of a
    small game hold empty ranges)."""
    games = small_batch(6, seed=41)
    p = np.random.default_rng(7).integers(-50, 51, size=(len(games), 4)).astype(np.int32)
    with eg.Batch(games, thresholds=4, scale=2, tail_rows=1, tail_sweeps=tail_sweeps,
                  tail_cluster=tail_cluster) as b:
        b.set_thresholds(p)
        _, st = b.solve()
        assert st.games_failed == 0 and st.tail_entries == len(games) * 4
        check_batch(b, games, p, 2)


@pytest.mark.parametrize("n,wmax,d,p", [
    (200, 3000, 400, [-900000, 0, 5000, 700000]),       # 32-bit credits, weights too large for a potential
    (200, 2600, 400, [-1000, 0, 7, 1000]),              # the largest weights that still have one
    (300, 20, 1 << 16, [-(1 << 19), 0, 3, 1 << 19]),    # 64-bit credits
    (2531, 100, 8, [473, -473, 0, 600]),                # several attempts: finite credits settle after 270 sweeps
])
def test_unit_certificates(n, wmax, d, p):
    g = workloads.cfg4_games(64)[62] if n == 2531 else eg.generate(4, n, 9, wmax, 90 + n, param=2)
    assert g.num_nodes == n
    games, thresholds = [g, g], np.array([p, p[::-1]], dtype=np.int32)
    with eg.Batch(games, thresholds=4, scale=d) as b:
        b.set_thresholds(thresholds)
        _, st = b.solve()
        assert st.games_failed == 0
        check_batch(b, games, thresholds, d)


def planned_units(edges, K, sms=148):
    """The units of a batch by the rule of its groups: halved from eight in games
    of more than 16,384 edges, to the least cost of a sweep that fits the SMs."""
    def cost(m, kg):
        return (m + 31) // 32 * {8: 34, 4: 22, 2: 12, 1: 7}[kg] // 2

    def group(m, limit):
        kg = 8
        while m > 16384 and kg > 1 and cost(m, kg) > limit:
            kg //= 2
        return kg

    limit = cost(16384, 8)
    while True:
        groups = [group(m, limit) for m in edges]
        count = sum(K // kg + (K % kg).bit_count() for kg in groups)
        if count <= sms or min(groups) == 8:
            return count
        limit += limit // 4


@pytest.mark.parametrize("num,nodes,K", [
    (3, 1024, 8), (3, 1025, 8), (3, 1900, 8), (3, 3000, 8), (3, 12000, 3),  # idle SMs
    (60, 4096, 8), (100, 1100, 8), (100, 2400, 8),                          # as many as fit
    (150, 1100, 5), (150, 2400, 5),                                         # more games than SMs
])
def test_groups_of_large_games(num, nodes, K):
    games = [eg.generate(4, nodes, 16, 20, 300 + i, param=2) for i in range(num)]
    rng = np.random.default_rng(num)
    p = rng.integers(-60, 61, size=(num, K)).astype(np.int32)
    got = []
    for group_max in (0, 8):
        with eg.Batch(games, thresholds=K, scale=4, group_max=group_max) as b:
            b.set_thresholds(p)
            _, st = b.solve()
            got.append((st.num_units, [b.credits(g) for g in range(num)]))
    assert got[0][0] == planned_units([g.num_edges for g in games], K)
    assert got[1][0] == num * (K // 8 + (K % 8).bit_count())
    for a, b in zip(got[0][1], got[1][1]):
        np.testing.assert_array_equal(a, b)


def chain(n, step=-1):
    """A path of n vertices into one that stays where it is at weight 0."""
    weight = np.full(n, step)
    weight[-1] = 0
    return eg.Game(row_ptr=np.arange(n + 1), succ=np.minimum(np.arange(1, n + 1), n - 1), weight=weight, num_nodes0=n // 2)


def test_time_limit_of_a_deep_game():
    """No vertex of the path is certified, and a kill phase takes them out one
    after the other: the limit must not wait for its end, and what the unit
    holds then are potentials, not credits."""
    n = 50_000
    with eg.Batch([chain(n)], thresholds=1, timeout_ms=20, park_percent=1000) as b:
        b.set_thresholds([0])
        b.solve(raise_on_error=False)  # loads the kernel
        status, st = b.solve(raise_on_error=False)
        assert st.games_failed == 1 and st.solve_ms < 60
        assert eg._ffi.STATUS_NAMES[b.game_result(0)[1]] == "EG_ERR_TIMEOUT"
        assert np.all(b.credits(0)[0] <= np.arange(n)[::-1])


def test_dropped_attempts_cost_no_more_than_the_sweeps():
    """Kill sweeps that run to their end on a path take four times the credit
    sweeps.  The second game has as many credit sweeps and short kills."""
    n = 16384
    deep, flat = chain(n), chain(n, 0)
    flat.weight[-2] = -5
    ms = []
    for g, want in ((deep, np.arange(n)[::-1]), (flat, np.where(np.arange(n) < n - 1, 5, 0))):
        with eg.Batch([g], thresholds=1, park_percent=1000) as b:
            b.set_thresholds([0])
            ms.append(min(b.solve()[1].solve_ms for _ in range(3)))
            np.testing.assert_array_equal(b.credits(0)[0], want)
    assert ms[0] < 3 * ms[1]


@pytest.mark.parametrize("group_max", [0, 1])
def test_a_group_in_which_some_thresholds_are_dropped(group_max):
    """A path at thresholds that leave its steps' cost (an attempt is dropped),
    take it away, and make every vertex unbounded (certified)."""
    n = 2000
    deep, zero, top = np.arange(n)[::-1], np.zeros(n, np.int64), np.full(n, eg.EG_TOP64)
    p, want = [0, -1, 1, 0, 7, -3, 0], [deep, zero, top, deep, top, zero, deep]
    with eg.Batch([chain(n)], thresholds=7, group_max=group_max) as b:
        b.set_thresholds(p)
        b.solve()
        np.testing.assert_array_equal(b.credits(0), np.array(want))


@pytest.mark.parametrize("levels,back", [(400, 0.01), (400, 0.3), (1500, 0.05)])
def test_deep_games_with_unbounded_parts(levels, back):
    """Groups whose thresholds are certified after different attempts, or dropped."""
    g, p = strip(levels, 4, back, levels), [0, 1, -1, 2, -2, 3, -8, 8]
    with eg.Batch([g], thresholds=8) as b:
        b.set_thresholds(p)
        b.solve()
        got = b.credits(0)
    for k, x in enumerate(p):
        np.testing.assert_array_equal(got[k], want(eg.threshold_game(g, x, 1)))
