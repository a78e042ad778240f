"""GPU tests of the frontier and dense rounds where default options take the
sweep solver: the round kinds are asked for, and the launches say that they
ran (a sweep solve is one launch)."""
from __future__ import annotations

import numpy as np
import pytest

import egsolver_b200 as eg
from egsolver_b200 import workloads
from oracle import oracle as O
from tests.conftest import to_top32
from tests.test_gpu_solver import DENSE_PATHS, big_weight_game, vid

pytestmark = pytest.mark.gpu

# the switch between round kinds at its default bounds, which, spelled out, ask for the rounds
SWITCH = dict(direction=eg.DIRECTION_SWITCH, dense_permille=40, sparse_permille=15)
DENSE = dict(direction=eg.DIRECTION_DENSE)
SPARSE = dict(direction=eg.DIRECTION_SPARSE)


def name(d):
    return vid(d) or "default"


@pytest.fixture(scope="module")
def cfg2_2e14():
    game = workloads.cfg2(1 << 14)
    return game, O.eg_solve(game, bits=64)[0]


@pytest.mark.parametrize("d", DENSE_PATHS, ids=name)
def test_data_paths_of_switching_rounds(cfg2_2e14, d):
    game, ref = cfg2_2e14
    f, st = eg.solve(game, credit_bits=64, **SWITCH, **d)
    np.testing.assert_array_equal(f, ref)
    assert st.kernel_launches > 1 and st.dense_rounds > 0
    assert st.credit_bits == (32 if d.get("narrow") else 64)


@pytest.mark.parametrize("d", [SWITCH, DENSE, dict(DENSE, wide_pairs=True)], ids=name)
def test_mg_near_the_32_bit_limit(d):
    game = big_weight_game()
    ref = O.eg_solve(game, bits=64)[0]
    f32, st = eg.solve(game, credit_bits=32, **d)
    assert st.kernel_launches > 1 and st.credit_bits == 32 and st.dense_rounds > 0
    np.testing.assert_array_equal(f32.astype(np.int64), to_top32(ref))
    f64, st = eg.solve(game, credit_bits=64, narrow=True, **d)
    assert st.credit_bits == 64
    np.testing.assert_array_equal(f64, ref)


@pytest.mark.parametrize("d", [SWITCH, SPARSE], ids=name)
@pytest.mark.parametrize("buckets", [dict(small_max_deg=2, large_min_deg=40), dict(small_max_deg=64, large_min_deg=65),
                                     dict(large_min_deg=9, task_edges=64)], ids=name)
@pytest.mark.parametrize("n", [1 << 12, 1 << 14])
def test_degree_buckets(n, buckets, d):
    game = workloads.cfg2(n)
    f, st = eg.solve(game, **d, **buckets)
    np.testing.assert_array_equal(f, O.eg_solve(game, bits=64)[0])
    assert st.kernel_launches > 1
    assert st.large_min_deg == buckets["large_min_deg"]


@pytest.mark.parametrize("d", [SWITCH, DENSE, SPARSE], ids=name)
def test_tuned_knobs(d):
    # of a shape that no other test tunes: the choice is cached by shape
    game = workloads.cfg2(1 << 13)
    ref = O.eg_solve(game, bits=64)[0]
    with eg.ResidentGame(game) as r:
        knobs, _ = r.tune(rounds=60, **d)
        _, st = r.solve(**d, **knobs)
        assert st.kernel_launches > 1
        np.testing.assert_array_equal(r.credits(64), ref)


# one CTA and the grid
@pytest.mark.parametrize("d", [SPARSE, SWITCH, DENSE], ids=name)
@pytest.mark.parametrize("n", [1000, 1 << 14])
def test_round_cap_cancel_and_time_limit(n, d):
    game = workloads.cfg2(n)
    ref = O.eg_solve(game, bits=64)[0]
    flag = eg.CancelFlag()
    try:
        with eg.ResidentGame(game) as r:
            status, st = r.solve(raise_on_error=False, max_rounds=2, **d)
            assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_LOOPCAP" and st.rounds == 2 and st.kernel_launches > 1
            part = r.credits()
            assert np.all(part <= ref) and np.any(part < ref)
            status, _ = r.solve(raise_on_error=False, timeout_ms=0.001, **d)
            assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_TIMEOUT"
            flag.set(1)
            status, st = r.solve(raise_on_error=False, cancel=flag, **d)
            assert eg._ffi.STATUS_NAMES[status] == "EG_ERR_CANCELLED" and st.rounds <= 2
            r.solve(**d)
            np.testing.assert_array_equal(r.credits(), ref)
    finally:
        flag.free()


@pytest.mark.parametrize("d", [SWITCH, SPARSE], ids=name)
def test_keep_layout(cfg2_2e14, d):
    game, ref = cfg2_2e14
    with eg.ResidentGame(game) as r:
        _, first = r.solve(**d)
        _, kept = r.solve(keep_layout=True, **d)
        np.testing.assert_array_equal(r.credits(), ref)
        r.solve(credit_bits=32, keep_layout=True, **d)
        np.testing.assert_array_equal(r.credits(32).astype(np.int64), to_top32(ref))
        assert 1 < kept.kernel_launches < first.kernel_launches - 20
        r.solve()  # the sweep solver in between
        r.solve(keep_layout=True, **d)
        np.testing.assert_array_equal(r.credits(), ref)


# large enough for the grid's kernels, whose dense rounds need the AUTO layout
@pytest.mark.parametrize("variant", [eg.VARIANT_WARP, eg.VARIANT_CTA])
def test_keep_layout_is_about_the_previous_solve(variant):
    game = eg.generate(4, 16000, 16, 20, 7, param=2)
    ref = O.eg_solve(game, bits=64)[0]
    assert game.num_edges > 1 << 17
    with eg.ResidentGame(game) as r:
        r.solve(variant=variant)
        np.testing.assert_array_equal(r.credits(), ref)
        r.solve()
        _, st = r.solve(keep_layout=True, **DENSE)
        np.testing.assert_array_equal(r.credits(), ref)
        assert st.dense_rounds > 0 and st.kernel_launches > 1
