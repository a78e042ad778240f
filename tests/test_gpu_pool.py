"""GPU tests of what calls share (eg_pool.cu): staged copies at the edges of
their chunks, threads that solve at once, and the transpose's device check."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import egsolver_b200 as eg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def csr(rng, rows, cols, nnz):
    rp = np.concatenate([[0], np.cumsum(np.bincount(rng.integers(0, rows, nnz), minlength=rows))]).astype(np.int64)
    return rp, rng.integers(0, cols, nnz).astype(np.int32), rng.integers(-9, 9, nnz).astype(np.int32)


# 131,072 entries of 4 bytes fill half a staging buffer
@pytest.mark.parametrize("nnz", [1, 65536, 65537, 131071, 131072, 131073, 2_300_003])
def test_staged_copies_of_the_transpose(nnz):
    rng = np.random.default_rng(nnz)
    rows, cols = 65535, 65537
    rp, col, val = csr(rng, rows, cols, nnz)
    for a, b in zip(eg.csr2csc(rows, cols, rp, col, val), O.csr2csc(rows, cols, rp, col, val)):
        np.testing.assert_array_equal(a, b)


def test_malformed_transposes_are_refused():
    rng = np.random.default_rng(2)
    rp, col, val = csr(rng, 3000, 2000, 40000)
    for bad_rp, bad_col in ((None, 2000), (None, -1), (1500, None)):
        r, c = rp.copy(), col.copy()
        if bad_col is not None:
            c[39999] = bad_col
        else:
            r[bad_rp] = 1 << 40
        with pytest.raises(eg.EGError) as ei:
            eg.csr2csc(3000, 2000, r, c, val)
        assert ei.value.name == "EG_ERR_INVALID"
    for a, b in zip(eg.csr2csc(3000, 2000, rp, col, val), O.csr2csc(3000, 2000, rp, col, val)):
        np.testing.assert_array_equal(a, b)


def test_threads_share_the_pools():
    """Games of several sizes solved by four threads at once, twice each."""
    games = [eg.generate(4, n, 16, 50, 5 + i, param=2) for i, n in enumerate((60, 900, 4000, 70000, 3000, 150))]
    alone = [eg.solve(g)[0] for g in games]
    wrong = []

    def work(k):
        for i in range(2 * len(games)):
            j = (i + k) % len(games)
            if not np.array_equal(eg.solve(games[j])[0], alone[j]):
                wrong.append(j)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("rows,cols,nnz,hot", [
    (1, 1, 1, 0), (5, 3, 2048, 0), (300, 7, 2049, 0),             # one CTA and two
    (100, 70000, 300, 0), (70000, 100, 300, 0), (1, 50000, 4000, 0),  # few entries, many columns or rows
    (3000, 4096, 60000, 2048), (3000, 4095, 60000, 20000),        # a column ordered here, one left to the sort
    (900, 1, 2500, 2500), (200003, 130001, 1500000, 9000), (250000, 300000, 900000, 200000),
])
def test_transpose_edges(rows, cols, nnz, hot):
    rng = np.random.default_rng(nnz)
    rp, col, val = csr(rng, rows, cols, nnz)
    if hot:
        col[rng.choice(nnz, hot, replace=False)] = cols - 1
    for a, b in zip(eg.csr2csc(rows, cols, rp, col, val), O.csr2csc(rows, cols, rp, col, val)):
        np.testing.assert_array_equal(a, b)


def test_a_lent_pointer_is_memory_of_its_own():
    """The array of credits_device can be mapped by other processes and peers
    (it is not the pool's), and freeing the game waits for work that another
    stream still has on it."""
    torch = pytest.importorskip("torch")
    from cuda.bindings import driver

    g = eg.generate(4, 3000, 16, 50, 9, param=2)
    r = eg.ResidentGame(g)
    for kw in (dict(credit_bits=64), dict(credit_bits=32), dict(credit_bits=64, direction=eg.DIRECTION_DENSE)):
        bits = kw["credit_bits"]
        r.solve(**kw)
        ptr, got_bits = r.credits_device()
        assert got_bits == bits
        err, legacy = driver.cuPointerGetAttribute(
            driver.CUpointer_attribute.CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE, ptr)
        assert err == driver.CUresult.CUDA_SUCCESS and legacy
        host = np.zeros(3000, np.int64 if bits == 64 else np.int32)
        assert driver.cuMemcpyDtoH(host.ctypes.data, ptr, host.nbytes)[0] == driver.CUresult.CUDA_SUCCESS
        np.testing.assert_array_equal(host, r.credits(bits))
    side = torch.cuda.Stream()
    done = torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(40_000_000)
        done.record()
    r.free()
    assert done.query()
