"""GPU tests of the sweep solver (eg_sweep.cu): exact credits where its
layout changes -- one CTA or the grid, values in shared or global memory,
edges staged or not, cut vertices -- and the hand-over to frontier rounds."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import egsolver_b200 as eg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hub_game(degrees, n=900, seed=5, wmax=40):
    """Vertices of out-degree 1..3 and one of each given out-degree, owners alternating."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(1, 4, n)
    deg[rng.choice(n, len(degrees), replace=False)] = degrees
    rp = np.concatenate([[0], np.cumsum(deg)])
    m = int(rp[-1])
    return eg.Game(row_ptr=rp, succ=rng.integers(0, n, m), weight=rng.integers(-wmax, wmax + 1, m),
                   owner=rng.integers(0, 2, n).astype(np.uint8))


def want(game):
    """The oracle's credits (it takes owner-sorted games)."""
    own = game.owners()
    order = np.argsort(own, kind="stable")
    inv = np.empty_like(order)
    inv[order] = np.arange(order.size)
    deg = np.diff(game.row_ptr)[order]
    idx = np.concatenate([np.arange(game.row_ptr[v], game.row_ptr[v + 1]) for v in order])
    g = eg.Game(row_ptr=np.concatenate([[0], np.cumsum(deg)]), succ=inv[game.succ[idx]], weight=game.weight[idx],
                num_nodes0=int((own == 0).sum()))
    f, st = O.eg_solve(g, bits=64, max_loop_=1 << 60)
    assert st["finished"]
    return f[inv]


# one CTA's shared memory ends between 3,000 and 3,700 vertices of out-degree 4
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1025, 3000, 3100, 3200, 3300, 3500, 3700])
def test_one_cta_and_grid_sizes(n):
    g = eg.generate(1, n, min(4, n), 9, 77 + n) if n > 4 else eg.Game(
        row_ptr=np.arange(n + 1), succ=np.arange(n)[::-1].copy(), weight=np.arange(n) - 1, num_nodes0=n // 2)
    f, st = eg.solve(g)
    np.testing.assert_array_equal(f, want(g))
    assert st.num_top == int((f == eg.EG_TOP64).sum())
    assert st.grid == 1 if n <= 3000 else st.grid in (1, 148)


@pytest.mark.parametrize("n,degrees", [(900, [255, 256, 257]), (900, [511, 513, 800]), (6000, [256, 4097, 5000]),
                                       (6000, [33] * 700)])
def test_cut_vertices(n, degrees):
    g = hub_game(degrees, n)
    ref = want(g)
    f, _ = eg.solve(g)
    np.testing.assert_array_equal(f, ref)
    f32, st = eg.solve(g, narrow=True)
    assert st.credit_bits == 32
    np.testing.assert_array_equal(f32, ref)


@pytest.fixture(scope="module")
def power_20k():
    g = eg.generate(2, 20000, 4096, 50, 11)
    return g, want(g)


# few CTAs: their values (28 B per vertex), then only their edges, leave shared memory
@pytest.mark.parametrize("ctas", [1, 3, 5, 147])
def test_values_and_edges_outside_shared_memory(power_20k, ctas):
    g, ref = power_20k
    f, st = eg.solve(g, grid_ctas=ctas)
    assert st.grid == ctas
    np.testing.assert_array_equal(f, ref)


@pytest.mark.parametrize("lanes_degree", [1, 2, 16, 40])
def test_lanes_per_vertex(lanes_degree):
    g = eg.generate(1, 6000, lanes_degree, 30, 3)
    f, _ = eg.solve(g)
    np.testing.assert_array_equal(f, want(g))


@pytest.mark.parametrize("n,n0,scale", [(9000, 0, 1), (9000, 9000, 1), (9000, 4000, 40000), (900, 500, 40000)])
def test_one_owner_and_wide_credits(n, n0, scale):
    """All vertices of one player (the other's parts are empty), and weights
    whose credits and potentials need 64 bits (the same game, scaled)."""
    g = eg.generate(4, n, 16, 100, 23, param=2)
    g = eg.Game(row_ptr=g.row_ptr, succ=g.succ, weight=g.weight, num_nodes0=n0)
    ref = want(g)
    f, _ = eg.solve(eg.Game(row_ptr=g.row_ptr, succ=g.succ, weight=g.weight * scale, num_nodes0=n0))
    np.testing.assert_array_equal(f, np.where(ref == eg.EG_TOP64, ref, ref * np.where(ref == eg.EG_TOP64, 1, scale)))


def test_least_weight():
    g = eg.Game(row_ptr=[0, 1, 2, 3], succ=[2, 2, 2], weight=[-(2**31), 2**31 - 1, 0], num_nodes0=1)
    f, st = eg.solve(g)
    np.testing.assert_array_equal(f, [2**31, 0, 0])
    assert st.mg == 2**31


def test_round_cap_on_the_grid_gives_a_lower_bound():
    g = eg.generate(4, 9000, 16, 100, 21, param=2)
    ref = want(g)
    with eg.ResidentGame(g) as r:
        status, st = r.solve(raise_on_error=False, max_rounds=1)
        assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_LOOPCAP" and st.rounds == 1
        part = r.credits()
        assert np.all(part <= ref) and np.any(part < ref)
        r.solve()
        np.testing.assert_array_equal(r.credits(), ref)


def test_hand_over_to_frontier_rounds():
    """Chains of 4,096 vertices along which one credit moves back a vertex
    per sweep: few raises in each of thousands of sweeps."""
    length, chains = 4096, 1100
    n = length * chains
    succ = np.arange(1, n + 1, dtype=np.int32)
    succ[length - 1::length] = np.arange(length - 1, n, length)
    weight = np.zeros(n, np.int32)
    weight[length - 2::length] = -5
    g = eg.Game(row_ptr=np.arange(n + 1), succ=succ, weight=weight, num_nodes0=n // 2)
    f, st = eg.solve(g)
    ref = np.full(n, 5)
    ref[length - 1::length] = 0
    np.testing.assert_array_equal(f, ref)
    assert st.rounds > 512 and st.num_top == 0


# on 37 CTAs 8 lanes share a vertex up to 2,368 vertices, 4 up to 4,736, 2 up
# to 9,472 (some parts differ by a vertex); complete digraphs whose edges fit
# 148 CTAs' shared memory, do but for a vertex each, and do not
@pytest.mark.parametrize("kind,n,deg,ctas", [(4, n, 16, 37) for n in (2000, 2368, 2400, 4736, 4800, 9400, 9700)] +
                         [(5, 3500, 30, 37), (1, 4000, 4, 37)] + [(3, n, n - 1, 0) for n in (1930, 2000, 2200)])
def test_lanes_that_share_a_vertex(kind, n, deg, ctas):
    g = eg.generate(kind, n, deg, 40, 5 + n, param=2 if kind == 4 else 6)
    f, st = eg.solve(g, grid_ctas=ctas)
    assert st.grid == (ctas or 148)
    np.testing.assert_array_equal(f, want(g))
    if g.num_edges < 50000:
        rng = np.random.default_rng(n)
        g = eg.Game(row_ptr=g.row_ptr, succ=g.succ, weight=g.weight * 40000, owner=rng.integers(0, 2, n).astype(np.uint8))
        f, _ = eg.solve(g, grid_ctas=ctas)
        np.testing.assert_array_equal(f, want(g))


def chain(n, step=-1):
    """One path of n vertices, the first half player 0's, into a vertex that
    stays where it is at weight 0: n - 1 steps of cost, no bound but the path's."""
    succ = np.minimum(np.arange(1, n + 1), n - 1)
    weight = np.full(n, step)
    weight[-1] = 0
    return eg.Game(row_ptr=np.arange(n + 1), succ=succ, weight=weight, num_nodes0=n // 2)


def test_time_limit_of_a_deep_game():
    """Of 400,000 vertices on a path none is certified, and a kill phase takes
    them out one after the other: the limit must not wait for its end."""
    n = 400_000
    with eg.ResidentGame(chain(n)) as r:
        r.solve(raise_on_error=False, max_rounds=1)  # loads the kernel
        status, st = r.solve(raise_on_error=False, timeout_ms=20)
        assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_TIMEOUT"
        assert st.solve_ms < 60
        assert np.all(r.credits() <= np.arange(n)[::-1])


def test_cancel_of_a_deep_game():
    n = 400_000
    flag = eg.CancelFlag()
    try:
        with eg.ResidentGame(chain(n)) as r:
            r.solve(raise_on_error=False, max_rounds=1)  # loads the kernel
            threading.Timer(0.02, flag.set).start()
            status, st = r.solve(raise_on_error=False, cancel=flag)
            assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_CANCELLED"
            assert st.solve_ms < 500  # of 2,000, or 3,700 with kills to their end
            assert np.all(r.credits() <= np.arange(n)[::-1])
    finally:
        flag.free()


# a path of 16,384 on the grid, a shorter one in one CTA
@pytest.mark.parametrize("n", [16384, 3000])
def test_dropped_attempts_cost_no_more_than_the_sweeps(n):
    """Kill sweeps that run to their end on a path take ten times the credit
    sweeps.  The second game has as many credit sweeps and short kills."""
    deep, flat = chain(n), chain(n, 0)
    flat.weight[-2] = -5
    with eg.ResidentGame(deep) as a, eg.ResidentGame(flat) as b:
        ms = [min(r.solve()[1].solve_ms for _ in range(3)) for r in (a, b)]
        np.testing.assert_array_equal(a.credits(), np.arange(n)[::-1])
        np.testing.assert_array_equal(b.credits(), np.where(np.arange(n) < n - 1, 5, 0))
    assert ms[0] < 4 * ms[1]


def chains(length, count, tops):
    """`count` paths of `length` vertices; a cost of 5 before the end of each,
    which moves back a vertex per sweep, or (the last `tops`) an end whose
    credit is unbounded, which does too."""
    n = length * count
    succ = np.arange(1, n + 1, dtype=np.int32)
    succ[length - 1::length] = np.arange(length - 1, n, length)
    weight = np.zeros(n, np.int32)
    weight[length - 2::length] = -5
    ref = np.full(n, 5)
    ref[length - 1::length] = 0
    if tops:
        weight[length * (count - tops) + length - 1::length] = -1
        ref[length * (count - tops):] = eg.EG_TOP64
    return eg.Game(row_ptr=np.arange(n + 1), succ=succ, weight=weight, num_nodes0=n // 2), ref


# long enough that the first look, at the end of the primal phase that passes
# 2,048 sweeps, finds raises in every path
@pytest.mark.parametrize("tops,narrow", [(0, False), (3, False), (3, True)])
def test_frontier_rounds_take_over(tops, narrow):
    g, ref = chains(16384, 260, tops)
    f, st = eg.solve(g, narrow=narrow)
    np.testing.assert_array_equal(f, ref)
    assert st.kernel_launches > 1 and st.pushes > 0 and 2048 <= st.dense_rounds < 16384
    assert st.num_top == tops * 16384 and st.credit_bits == (32 if narrow else 64)


def test_round_cap_after_the_hand_over():
    g, ref = chains(16384, 260, 1)
    with eg.ResidentGame(g) as r:
        status, st = r.solve(raise_on_error=False, max_rounds=7000)
        assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_LOOPCAP"
        assert st.rounds == 7000 and st.pushes > 0
        part = r.credits()
        assert np.all(part <= ref) and np.any(part < ref) and np.any(part == 5)


def test_hand_over_without_memory_for_it():
    """The frontier rounds' arrays do not fit: the sweeps end the solve."""
    torch = pytest.importorskip("torch")
    g, ref = chains(8192, 520, 2)
    with eg.ResidentGame(g) as r:
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
        try:
            status, st = r.solve(raise_on_error=False)
        finally:
            del hog
            torch.cuda.empty_cache()
        assert status == 0 and st.pushes == 0 and st.kernel_launches == 2
        np.testing.assert_array_equal(r.credits(), ref)
        _, st = r.solve()
        assert st.pushes > 0
        np.testing.assert_array_equal(r.credits(), ref)


def test_knobs_of_the_rounds_leave_the_sweep_solver_alone():
    """dense_sweeps is a knob of the dense rounds, and one the tuner sets: the
    sweep solver runs two sweeps between its barriers whatever it says."""
    g = eg.generate(4, 9000, 16, 100, 21, param=2)
    f, st = eg.solve(g)
    for k in (1, 2, 4):
        f1, st1 = eg.solve(g, dense_sweeps=k)
        np.testing.assert_array_equal(f1, f)
        assert st1.grid == st.grid > 1 and st1.rounds < st1.dense_rounds


def strip(levels, width, back, seed):
    """Levels of `width` vertices, two edges of cost 1 to 3 from each to the
    next level, the last level at rest; a share `back` of the vertices has a
    third edge to some earlier level, which gains or costs a little."""
    rng = np.random.default_rng(seed)
    n = levels * width
    rows = []
    for v in range(n):
        lv = v // width
        if lv == levels - 1:
            rows.append([(v, 0)])
            continue
        e = [((lv + 1) * width + int(rng.integers(width)), -int(rng.integers(1, 4))) for _ in range(2)]
        if rng.random() < back:
            e.append((int(rng.integers(v + 1)), int(rng.integers(-3, 40))))
        rows.append(e)
    return eg.Game(row_ptr=np.concatenate([[0], np.cumsum([len(e) for e in rows])]),
                   succ=np.array([s for e in rows for s, _ in e]), weight=np.array([w for e in rows for _, w in e]),
                   owner=rng.integers(0, 2, n).astype(np.uint8))


# one CTA and the grid; attempts that are dropped, then some that certify
@pytest.mark.parametrize("levels,width", [(500, 4), (2000, 4)])
@pytest.mark.parametrize("back", [0.01, 0.05, 0.3])
def test_deep_games_with_unbounded_parts(levels, width, back):
    g = strip(levels, width, back, levels)
    f, st = eg.solve(g)
    assert (st.grid > 1) == (levels > 500)
    np.testing.assert_array_equal(f, want(g))


# one CTA and the grid; the last of a slice, of a player, of the game
@pytest.mark.parametrize("n,sink", [(100, 0), (100, 63), (3000, 2999), (6000, 31), (20000, 9999), (20000, 19999)])
def test_device_games_with_a_sink_are_refused(n, sink):
    """A game that is on the device already has not been through the host's checks."""
    torch = pytest.importorskip("torch")
    g = eg.generate(1, n, 4, 9, n + sink)
    deg = np.full(n, 4)
    for counts in (np.where(np.arange(n) == sink, 0, deg), deg):
        rp = np.concatenate([[0], np.cumsum(counts)])
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rp, g.succ, g.weight)]
        torch.cuda.synchronize()
        r = eg.ResidentGame.from_device(n, int(rp[-1]), g.num_nodes0, *(x.data_ptr() for x in dev))
        if counts is deg:
            r.solve()
            np.testing.assert_array_equal(r.credits(), want(g))
        else:
            with pytest.raises(eg.EGError) as ei:
                r.solve()
            assert ei.value.name == "EG_ERR_INVALID"
        r.free()
