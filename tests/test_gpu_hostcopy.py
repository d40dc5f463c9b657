"""Pageable arrays through the page-locked pieces, which exist only once a
process has copied 64 MiB directly: the fixture makes that traffic and keeps a
context that holds the pieces."""
import ctypes as C
import threading

import numpy as np
import pytest

import dsgdpp_b200 as P

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _staged():
    fn = P.lib.dsgdpp_staged_bytes
    fn.restype = C.c_uint64
    return fn()


def _lock(a):
    import torch
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a
                            ).pin_memory().numpy().view(a.dtype)


def _config(m, n, r, **kw):
    return P.Config(m=m, n=n, rank=r, d=1, precision="fp64", **kw)


@pytest.fixture(scope="module")
def pieces():
    m = 40 * MB // 8
    with P.Context(_config(m, 2, 1)) as holder:
        before = _staged()
        for _ in range(3):
            holder.set_factors(np.zeros((m, 1)), np.zeros((2, 1)))
        assert _staged() - before >= m * 8
        yield


# rows of W of 8 bytes: the bytes of W in 8ths
@pytest.mark.parametrize("m,staged", [
    (6 * MB // 8 - 1, False), (6 * MB // 8, True), (6 * MB // 8 + 1, True), (7 * MB // 8, True),
    (16 * MB // 8, True), (17 * MB // 8 - 1, True), (33 * MB // 8 + 5, True)])
def test_factors_of_every_split_into_pieces(pieces, m, staged):
    rng = np.random.default_rng(m)
    W0, H0 = rng.standard_normal((m, 1)), rng.standard_normal((3, 1))
    with P.Context(_config(m, 3, 1)) as ctx:
        for give, through in ((np.copy, staged), (_lock, False)):
            at = _staged()
            ctx.set_factors(give(W0), give(H0))
            assert _staged() - at == (m * 8 if through else 0)
            W, H = give(np.zeros_like(W0)), give(np.zeros_like(H0))
            at = _staged()
            ctx.get_factors_into(W, H)
            assert _staged() - at == (m * 8 if through else 0)
            np.testing.assert_array_equal(W, W0)
            np.testing.assert_array_equal(H, H0)


@pytest.mark.parametrize("nnz", [786_431, 786_433, 1_572_865, 2_000_003])
def test_matrix_through_pieces_and_page_locked(pieces, nnz):
    rng = np.random.default_rng(nnz)
    rows = rng.integers(0, 5000, nnz).astype(np.uint32)  # some pairs repeat: values are summed
    cols = rng.integers(0, 4000, nnz).astype(np.uint32)
    vals = rng.standard_normal(nnz)
    W0, H0 = rng.standard_normal((5000, 4)), rng.standard_normal((4000, 4))
    sizes = [b for b in (4 * nnz, 4 * nnz, 8 * nnz) if b >= 6 * MB]
    got = []
    for give in (np.copy, _lock):
        with P.Context(P.Config(m=5000, n=4000, rank=4, d=3, precision="fp64")) as ctx:
            at = _staged()
            ctx.set_matrix(P.TRAIN, give(rows), give(cols), give(vals))
            assert _staged() - at == (sum(sizes) if give is np.copy else 0)
            ctx.set_factors(W0, H0)
            got.append((ctx.block_nnz(), *ctx.nnz12()[:2], ctx.nzsl(P.TRAIN)))
            bad = rows.copy()
            bad[nnz // 2] = 5000  # refused while the values are still on their way
            with pytest.raises(P.DsgdppError):
                ctx.set_matrix(P.TRAIN, give(bad), give(cols), give(vals))
            ctx.set_matrix(P.TRAIN, give(rows), give(cols), give(vals))
            assert ctx.nzsl(P.TRAIN) == got[-1][-1]
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("threads", [2, 5])  # five copies at once want more pieces than there are
def test_contexts_on_several_threads_share_the_pieces(pieces, threads):
    m, errors = 20 * MB // 8 + 3, []

    def one(k):
        try:
            rng = np.random.default_rng(k)
            with P.Context(_config(m, 2, 1)) as ctx:
                H0 = rng.standard_normal((2, 1))
                for _ in range(6):
                    W0 = rng.standard_normal((m, 1))
                    ctx.set_factors(W0, H0)
                    W, H = ctx.get_factors()
                    np.testing.assert_array_equal(W, W0)
                    np.testing.assert_array_equal(H, H0)
        except BaseException as e:  # reported by the test's own thread
            errors.append(e)

    at = _staged()
    pool = [threading.Thread(target=one, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not errors, errors[0]
    assert _staged() > at
