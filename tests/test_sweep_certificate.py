"""CPU model of the sweep solver's certificate (eg_sweep.cu): a set that its
kill sweeps leave is TOP in the oracle's solution, whatever numbers the
potentials are, and its schedule ends at the oracle's credits."""
from __future__ import annotations

import numpy as np

import egsolver_b200 as eg
from oracle import oracle as O

TOP, LOW = 1 << 62, -(1 << 62)


def minmax(g, v):
    own, rp = g.owners(), g.row_ptr[:-1]
    return np.where(own == 0, np.minimum.reduceat(v, rp), np.maximum.reduceat(v, rp)), np.where(
        own == 0, np.maximum.reduceat(v, rp), np.minimum.reduceat(v, rp))


def primal(g, f, mg):
    x = minmax(g, f[g.succ] - g.weight.astype(np.int64))[0]
    return np.maximum(f, np.where(x > mg, TOP, np.maximum(x, 0)))


def dual_lift(g, d, shift):
    return np.maximum(minmax(g, d[g.succ] + (g.weight.astype(np.int64) << shift) + 1)[1], 0)


def certified(g, f, d, shift):
    k = np.where(f == TOP, LOW, d)
    while True:
        out = (k != LOW) & (k != TOP) & (dual_lift(g, k, shift) > k)
        if not out.any():
            return (k != LOW) & (k != TOP)
        k = np.where(out, TOP, k)


def games():
    for seed in range(40):
        kind, deg = [(1, 3), (2, 40), (4, 9), (5, 20)][seed % 4]
        yield eg.generate(kind, 50 + 13 * seed, deg, 1 + 3 * (seed % 7), 600 + seed, param=2 if kind == 4 else 5)


def test_certificates_are_sound_for_any_potentials():
    rng = np.random.default_rng(8)
    found = 0
    for g in games():
        ref = O.eg_solve(g, bits=64)[0]
        f, mg = np.zeros(g.num_nodes, np.int64), eg.compute_mg(g)
        for shift in (0, 3, 11):
            d = np.zeros(g.num_nodes, np.int64)
            for _ in range(6):
                s = certified(g, f, d, shift)
                assert np.all(ref[s] == O.TOP64)
                found += int(s.sum())
                d = np.maximum(d, dual_lift(g, d, shift)) + rng.integers(0, 3, d.size) * (shift == 3)
                d = np.where(d > 1 << 61, TOP, d)
            f = primal(g, f, mg)
    assert found > 1000


def test_schedule_ends_at_the_oracles_credits():
    for g in games():
        ref = O.eg_solve(g, bits=64)[0]
        n, mg = g.num_nodes, eg.compute_mg(g)
        f, d, length, shift = np.zeros(n, np.int64), np.zeros(n, np.int64), 4, min(20, int(n).bit_length())
        while True:
            raised = True
            for _ in range(length):
                new = primal(g, f, mg)
                raised = bool((new != f).any())
                f = new
                if not raised:
                    break
            if not raised:
                break
            d = np.where(f == TOP, LOW, d)
            for _ in range(8):
                y = dual_lift(g, d, shift)
                d = np.where((d == LOW) | (d == TOP) | (y <= d), d, np.where(y > 1 << 61, TOP, y))
            f = np.where(certified(g, f, d, shift), TOP, f)
            length = min(2 * length, 64)
        np.testing.assert_array_equal(np.where(f == TOP, O.TOP64, f), ref)
