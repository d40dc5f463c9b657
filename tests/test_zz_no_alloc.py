"""The allocation-free loss entry point (dsgdpp_nzsl_fp32_noalloc).

Some callers cannot allocate device memory themselves -- code that runs inside
another framework's memory pool, or under an allocator it does not own -- so
this entry point takes caller-owned device buffers and keeps its scratch in a
fixed device array.  This test calls it through the C ABI and checks its
result against the existing entry point (dsgdpp_nzsl on a context holding the
same FP32 data), within the 1e-12 relative tolerance of the other loss tests,
on consecutive calls that share the scratch.  It lives in a file of its own
that pytest collects last.
"""
import ctypes as C

import numpy as np
import pytest

import dsgdpp_b200 as P
from dsgdpp_b200 import synth

pytestmark = pytest.mark.gpu
LOSS_RTOL = 1e-12


def _device(torch, a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def _padded(torch, a, ld):
    out = np.zeros((a.shape[0], ld), np.float32)
    out[:, :a.shape[1]] = a.astype(np.float32)
    return _device(torch, out, torch.float32)


def _call(torch, rows, cols, vals, W, H, r, ld, partials=0):
    out = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    rc = P.lib.dsgdpp_nzsl_fp32_noalloc(
        rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), vals.numel(), W.data_ptr(),
        H.data_ptr(), r, ld, partials, out.data_ptr(), None)
    assert rc == P.OK
    torch.cuda.synchronize()
    return float(out.item())


def test_noalloc_nzsl_matches_context_loss():
    import torch
    r, ld = 30, 32
    p = synth.make(3000, 2000, 80000, 9000, rank_true=8, r=r, noise=0.1, seed=21, kind="zipf")
    with P.Context(P.Config(m=p.m, n=p.n, rank=r, d=4, precision="fp32")) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
        ctx.set_factors(p.W0, p.H0)
        want_train, want_test = ctx.nzsl(P.TRAIN), ctx.nzsl(P.TEST)
    W, H = _padded(torch, p.W0, ld), _padded(torch, p.H0, ld)
    # entry values are held in FP32, as in the context
    tr = [_device(torch, p.rows.view(np.int32), torch.int32),
          _device(torch, p.cols.view(np.int32), torch.int32),
          _device(torch, p.vals.astype(np.float32), torch.float32)]
    te = [_device(torch, p.trows.view(np.int32), torch.int32),
          _device(torch, p.tcols.view(np.int32), torch.int32),
          _device(torch, p.tvals.astype(np.float32), torch.float32)]
    # two calls in a row share the scratch: training entries, then test entries
    got_train = _call(torch, *tr, W, H, r, ld)
    got_test = _call(torch, *te, W, H, r, ld)
    assert got_train == pytest.approx(want_train, rel=LOSS_RTOL)
    assert got_test == pytest.approx(want_test, rel=LOSS_RTOL)
    # fewer partial sums than the previous call: stale slots are not read
    assert _call(torch, *te, W, H, r, ld, partials=7) == pytest.approx(want_test, rel=LOSS_RTOL)
    assert _call(torch, *tr, W, H, r, ld, partials=4096) == pytest.approx(
        want_train, rel=LOSS_RTOL)


def test_noalloc_rejects_requests_beyond_capacity():
    import torch
    W = torch.zeros((4, 4), dtype=torch.float32, device="cuda")
    idx = torch.zeros(1, dtype=torch.int32, device="cuda")
    v = torch.zeros(1, dtype=torch.float32, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    args = (idx.data_ptr(), idx.data_ptr(), v.data_ptr(), 1, W.data_ptr(), W.data_ptr(), 4, 4)
    assert P.lib.dsgdpp_nzsl_fp32_noalloc(*args, 4097, out.data_ptr(), None) == P.E_INVALID
    # a row stride that is not a whole number of 16-byte vectors is refused
    assert P.lib.dsgdpp_nzsl_fp32_noalloc(idx.data_ptr(), idx.data_ptr(), v.data_ptr(), 1,
                                          W.data_ptr(), W.data_ptr(), 3, 3, 0, out.data_ptr(),
                                          None) == P.E_INVALID
    # a row wider than the widest loss kernel (512 floats) is refused, not failed
    wide = torch.zeros((2, 516), dtype=torch.float32, device="cuda")
    assert P.lib.dsgdpp_nzsl_fp32_noalloc(idx.data_ptr(), idx.data_ptr(), v.data_ptr(), 1,
                                          wide.data_ptr(), wide.data_ptr(), 516, 516, 0,
                                          out.data_ptr(), None) == P.E_INVALID
    assert P.lib.dsgdpp_nzsl_fp32_noalloc(*args, 1, out.data_ptr(), None) == P.OK
    torch.cuda.synchronize()


@pytest.mark.parametrize("r,ld,shift", [(30, 32, 0), (30, 32, 4), (32, 32, 4), (8, 16, 0),
                                        (5, 24, 4), (7, 12, 0), (100, 512, 4)])
def test_noalloc_leaves_padding_and_alignment_to_the_caller(r, ld, shift):
    # rows on 16 but not 32 bytes, and a padding that holds anything
    import torch
    p = synth.make(300, 200, 2011, 10, rank_true=5, r=r, noise=0.1, seed=r)
    def rows_of(a):
        flat = np.full(shift + a.shape[0] * ld, np.nan, np.float32)
        flat[shift:].reshape(a.shape[0], ld)[:, :r] = a
        return _device(torch, flat, torch.float32)[shift:]
    W, H = rows_of(p.W0), rows_of(p.H0)
    got = _call(torch, _device(torch, p.rows.view(np.int32), torch.int32),
                _device(torch, p.cols.view(np.int32), torch.int32),
                _device(torch, p.vals, torch.float32), W, H, r, ld)
    f = lambda a: a.astype(np.float32).astype(np.float64)
    want = np.sum((f(p.vals) - np.einsum("ij,ij->i", f(p.W0)[p.rows], f(p.H0)[p.cols])) ** 2)
    assert got == pytest.approx(float(want), rel=LOSS_RTOL)


@pytest.mark.parametrize("nnz", [1, 31, 33, 2000])
def test_noalloc_reads_only_the_rows_that_entries_name(nnz):
    # the bases point 1000 rows before the callers' memory, as those of a part
    # of a larger matrix do
    import torch
    r, ld, first = 30, 32, 1000
    p = synth.make(300, 200, 4000, 10, rank_true=5, r=r, noise=0.1, seed=nnz)
    W, H = _padded(torch, p.W0, ld), _padded(torch, p.H0, ld)
    rows, cols, vals = p.rows[:nnz], p.cols[:nnz], p.vals[:nnz]
    out = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    dr = _device(torch, (rows + np.uint32(first)).view(np.int32), torch.int32)
    dc = _device(torch, (cols + np.uint32(first)).view(np.int32), torch.int32)
    dv = _device(torch, vals, torch.float32)
    back = first * ld * 4
    assert P.lib.dsgdpp_nzsl_fp32_noalloc(
        dr.data_ptr(), dc.data_ptr(), dv.data_ptr(), nnz, W.data_ptr() - back,
        H.data_ptr() - back, r, ld, 0, out.data_ptr(), None) == P.OK
    torch.cuda.synchronize()
    f = lambda a: a.astype(np.float32).astype(np.float64)
    want = np.sum((f(vals) - np.einsum("ij,ij->i", f(p.W0)[rows], f(p.H0)[cols])) ** 2)
    assert float(out.item()) == pytest.approx(float(want), rel=LOSS_RTOL)


def test_noalloc_calls_of_any_rank_are_captured_after_the_first_call():
    import torch
    p = synth.make(300, 200, 2000, 10, rank_true=5, r=200, noise=0.1, seed=3)
    ids = [_device(torch, a.view(np.int32), torch.int32) for a in (p.rows, p.cols)]
    v = _device(torch, p.vals, torch.float32)
    W, H = _padded(torch, p.W0, 200), _padded(torch, p.H0, 200)
    want = [_call(torch, *ids, v, W, H, 20, 200)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st = torch.cuda.current_stream().cuda_stream
        for k, r in enumerate((20, 200)):  # the two lengths of rows
            assert P.lib.dsgdpp_nzsl_fp32_noalloc(
                *[a.data_ptr() for a in (*ids, v)], v.numel(), W.data_ptr(), H.data_ptr(), r, 200,
                0, out[k:].data_ptr(), st) == P.OK
    graph.replay()
    torch.cuda.synchronize()
    want.append(_call(torch, *ids, v, W, H, 200, 200))
    assert out.tolist() == want


@pytest.mark.parametrize("r,ld", [(66, 68), (98, 100), (130, 132), (250, 252), (258, 260),
                                  (378, 380), (450, 452), (135, 136), (253, 256), (381, 384),
                                  (511, 512)])
def test_noalloc_masks_the_padding_in_every_mapping_of_eight_lanes_and_more(r, ld):
    test_noalloc_leaves_padding_and_alignment_to_the_caller(r, ld, 0)
