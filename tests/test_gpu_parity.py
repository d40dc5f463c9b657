"""GPU parity tests: the CUDA path (through the C ABI) against the CPU oracle.

Tolerances:
* FP64 replay factors: bit-identical to the oracle (the bar is 1e-10 relative
  per entry; the replay repeats every operation in the reference order);
* FP64 losses: 1e-12 relative (the terms are identical, only the summation
  order differs);
* blocking, counts, schedules: exact;
* FP32 / BF16 Hogwild runs: final test RMSE within a stated tolerance of the
  FP64 oracle's, since updates inside a block run concurrently.
"""
import numpy as np
import pytest

import dsgdpp_b200 as P
from dsgdpp_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LOSS_RTOL = 1e-12


def _problem(m=500, n=400, nnz=6000, ntest=600, r=10, seed=5, kind="uniform"):
    return synth.make(m, n, nnz, ntest, rank_true=min(r, 8), r=r, noise=0.1, seed=seed,
                      kind=kind)


def _pair(p, r, d, precision="fp64", exec="replay", launch="stream", **kw):
    okw = {k: v for k, v in kw.items() if k in ("update", "update_lambda", "regularize",
                                                 "regularize_lambda", "loss", "loss_lambda",
                                                 "truncate", "sgd_order", "stratum_order")}
    ref = O.Problem(p.m, p.n, r, d, p.rows, p.cols, p.vals, p.trows, p.tcols, p.tvals)
    ref.configure(**okw)
    ref.set_factors(p.W0, p.H0)
    cfg = P.Config(m=p.m, n=p.n, rank=r, d=d, precision=precision, exec=exec, launch=launch,
                   **{k: v for k, v in kw.items()})
    ctx = P.Context(cfg)
    ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
    ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
    ctx.set_factors(p.W0, p.H0)
    return ref, ctx


@pytest.mark.parametrize("update", ["Nzsl", "Nzsl_L2", "Nzsl_Nzl2"])
@pytest.mark.parametrize("sgd_order", ["SEQ", "WR", "WOR"])
@pytest.mark.parametrize("truncate", [None, (-0.3, 0.3)])
def test_replay_bit_exact(update, sgd_order, truncate):
    p = _problem()
    d = 3
    ref, ctx = _pair(p, 10, d, update=update, update_lambda=0.5, sgd_order=sgd_order,
                     truncate=truncate, loss="Nzsl")
    with ctx:
        R = P.Random32(77)
        for _ in range(2):
            sched, seeds = P.draw_schedule(R, d, "COWOR")
            ctx.epoch_explicit(0.02, sched, seeds)
            ref.epoch_explicit(0.02, sched, seeds)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


@pytest.mark.parametrize("r", [1, 3, 32, 33, 64, 128])
def test_replay_ranks(r):
    p = _problem(m=300, n=200, nnz=3000, r=r)
    d = 2
    ref, ctx = _pair(p, r, d)
    with ctx:
        sched, seeds = P.draw_schedule(P.Random32(r), d, "WOR")
        ctx.epoch_explicit(0.01, sched, seeds)
        ref.epoch_explicit(0.01, sched, seeds)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


def test_replay_l2_regularize_exact():
    p = _problem()
    d = 4
    ref, ctx = _pair(p, 10, d, update="Nzsl", regularize="L2", regularize_lambda=0.05,
                     loss="Nzsl_L2", loss_lambda=0.05)
    with ctx:
        R = P.Random32(3)
        for _ in range(2):
            sched, seeds = P.draw_schedule(R, d, "COWOR")
            ctx.epoch_explicit(0.05, sched, seeds)
            ref.epoch_explicit(0.05, sched, seeds)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


@pytest.mark.parametrize("stratum_order", ["SEQ", "RSEQ", "WR", "WOR", "COWOR"])
def test_replay_master_rng_epochs(stratum_order):
    # dsgdpp_epoch draws the schedule itself, like DsgdPpRunner::epoch
    p = _problem()
    d = 2
    ref, ctx = _pair(p, 10, d, stratum_order=stratum_order)
    with ctx:
        ctx.seed(1499881717)
        ref.seed(1499881717)
        for _ in range(3):
            ctx.epoch(0.01)
            ref.epoch(0.01)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


@pytest.mark.parametrize("loss", ["Nzsl", "Nzsl_L2", "Nzsl_Nzl2"])
def test_loss_parity(loss):
    p = _problem(m=2000, n=1500, nnz=60000, ntest=5000, r=16)
    ref, ctx = _pair(p, 16, 4, loss=loss, loss_lambda=0.3)
    with ctx:
        assert ctx.loss() == pytest.approx(ref.loss(), rel=LOSS_RTOL)
        assert ctx.nzsl(P.TEST) == pytest.approx(ref.nzsl(1), rel=LOSS_RTOL)
        assert ctx.nzsl(P.TRAIN) == pytest.approx(ref.nzsl(0), rel=LOSS_RTOL)
        for a, b in zip(ctx.l2(), ref.l2()):
            assert a == pytest.approx(b, rel=LOSS_RTOL)
        for a, b in zip(ctx.nzl2(), ref.nzl2()):
            assert a == pytest.approx(b, rel=LOSS_RTOL)


def test_loss_parity_fp32_and_bf16_factors():
    # the FP64 loss of stored low-precision factors equals the oracle's loss of
    # the same factors read back as doubles
    p = _problem(m=2000, n=1500, nnz=40000, r=32)
    # FP32 / BF16 factor storage keeps the entry values in FP32 (12-byte records)
    p.vals = p.vals.astype(np.float32).astype(np.float64)
    p.tvals = p.tvals.astype(np.float32).astype(np.float64)
    for prec in ("fp32", "bf16"):
        ref, ctx = _pair(p, 32, 4, precision=prec, exec="hogwild")
        with ctx:
            W, H = ctx.get_factors()
            ref.set_factors(W, H)
            assert ctx.nzsl(P.TRAIN) == pytest.approx(ref.nzsl(0), rel=LOSS_RTOL)
            assert ctx.loss() == pytest.approx(ref.loss(), rel=LOSS_RTOL)


def _extreme(rng, shape):
    """Factor values over the whole float range: zeros, subnormals, tiny,
    ordinary and large magnitudes, both signs."""
    kind = rng.choice(5, size=shape, p=[0.2, 0.1, 0.1, 0.58, 0.02])
    mag = np.select([kind == 0, kind == 1, kind == 2, kind == 3, kind == 4],
                    [0.0, rng.uniform(1e-42, 1e-39, shape), rng.uniform(1e-22, 1e-18, shape),
                     rng.uniform(0.0, 2.0, shape), rng.uniform(1e3, 1e4, shape)])
    return mag * rng.choice([-1.0, 1.0], size=shape)


@pytest.mark.parametrize("r", [7, 32, 100])
def test_loss_parity_extreme_factor_values(r):
    # the FP32/BF16 loss kernels form exact FP64 products (H's values built
    # from their bits, scaled by a power of two and back): zeros, subnormal,
    # tiny and large factor values give the oracle's loss of the same stored
    # factors, at ranks with and without a partial last vector
    p = _problem(m=300, n=200, nnz=6000, ntest=500, r=r)
    p.vals = p.vals.astype(np.float32).astype(np.float64)
    p.tvals = p.tvals.astype(np.float32).astype(np.float64)
    rng = np.random.default_rng(r)
    p.W0 = _extreme(rng, p.W0.shape)
    p.H0 = _extreme(rng, p.H0.shape)
    for prec in ("fp32", "bf16"):
        ref, ctx = _pair(p, r, 4, precision=prec, exec="hogwild")
        with ctx:
            W, H = ctx.get_factors()
            assert np.count_nonzero((W != 0) & (np.abs(W) < 1.1754944e-38)) > 0  # subnormals stored
            ref.set_factors(W, H)
            assert ctx.nzsl(P.TRAIN) == pytest.approx(ref.nzsl(0), rel=LOSS_RTOL)
            assert ctx.nzsl(P.TEST) == pytest.approx(ref.nzsl(1), rel=LOSS_RTOL)
            assert ctx.loss() == pytest.approx(ref.loss(), rel=LOSS_RTOL)


def test_blocking_and_counts():
    p = _problem(m=1001, n=997, nnz=20000, kind="zipf")
    for d in (1, 3, 8):
        ref, ctx = _pair(p, 8, d)
        with ctx:
            np.testing.assert_array_equal(ctx.block_nnz(P.TRAIN), ref.block_nnz(0))
            np.testing.assert_array_equal(ctx.block_nnz(P.TEST), ref.block_nnz(1))
            a, b, mx = ctx.nnz12()
            ra, rb, rmx = ref.nnz12()
            np.testing.assert_array_equal(a, ra)
            np.testing.assert_array_equal(b, rb)
            assert mx == rmx


def test_duplicates_are_summed():
    rows = np.array([5, 0, 5, 3, 0, 5], np.uint32)
    cols = np.array([1, 7, 1, 2, 0, 1], np.uint32)
    vals = np.array([1.0, 2.0, 0.5, 3.0, 4.0, 0.25])
    W0 = np.random.default_rng(0).uniform(-0.5, 0.5, (6, 2))
    H0 = np.random.default_rng(1).uniform(-0.5, 0.5, (8, 2))
    ref = O.Problem(6, 8, 2, 2, rows, cols, vals).configure()
    ref.set_factors(W0, H0)
    with P.Context(P.Config(m=6, n=8, rank=2, d=2, precision="fp64", exec="replay")) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        np.testing.assert_array_equal(ctx.block_nnz(), ref.block_nnz())
        assert ctx.nzsl() == pytest.approx(ref.nzsl(), rel=LOSS_RTOL)


@pytest.mark.parametrize("layout", ["shuffled", "col_runs", "row_runs"])
def test_hogwild_layouts_block_and_merge_like_the_oracle(layout):
    """Hogwild training records are blocked and laid out by one sort whose key
    permutes the positions inside a block.  On a matrix where nearly every
    position of every block holds one or more entries (uneven block extents,
    so the permuted ranges are not powers of two), two positions sharing a key
    would merge distinct entries: the block counts and the training loss must
    still equal the oracle's, which merges exact duplicates only
    (ReadMatrixBlocksMm's coordinate sort, mf/matrix/io/read_impl.h:162-164)."""
    rng = np.random.default_rng(3)
    m, n, d, r = 203, 181, 3, 5
    rows = rng.integers(0, m, 150000).astype(np.uint32)
    cols = rng.integers(0, n, 150000).astype(np.uint32)
    vals = rng.normal(0, 1, 150000)
    W0 = rng.uniform(-0.5, 0.5, (m, r))
    H0 = rng.uniform(-0.5, 0.5, (n, r))
    ref = O.Problem(m, n, r, d, rows, cols, vals).configure()
    ref.set_factors(W0, H0)
    assert len(set(zip(rows.tolist(), cols.tolist()))) > 0.98 * m * n
    cfg = P.Config(m=m, n=n, rank=r, d=d, precision="fp64", exec="hogwild", layout=layout)
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        np.testing.assert_array_equal(ctx.block_nnz(), ref.block_nnz())
        assert ctx.nzsl() == pytest.approx(ref.nzsl(), rel=LOSS_RTOL)


def test_run_trace_matches_oracle():
    p = _problem(m=800, n=600, nnz=10000, ntest=1000)
    ref, ctx = _pair(p, 10, 2)
    with ctx:
        ctx.seed(42)
        ref.seed(42)
        tr = ctx.run(6, "BoldDriver", 0.01)
        rt = ref.run(6, "BoldDriver", 0.01)
        for k, row in enumerate(tr):
            assert row["loss"] == pytest.approx(rt[k, 0], rel=LOSS_RTOL)
            assert row["test_loss"] == pytest.approx(rt[k, 1], rel=LOSS_RTOL)
            if k:
                assert row["eps"] == rt[k, 2]


def test_empty_matrix_and_empty_blocks():
    p = _problem(m=50, n=40, nnz=30, ntest=0)
    ref, ctx = _pair(p, 4, 4)  # 4 x 8 blocks, most of them empty
    with ctx:
        sched, seeds = P.draw_schedule(P.Random32(1), 4, "COWOR")
        ctx.epoch_explicit(0.1, sched, seeds)
        ref.epoch_explicit(0.1, sched, seeds)
        np.testing.assert_array_equal(ctx.get_factors()[0], ref.get_factors()[0])
        assert ctx.nzsl(P.TEST) == 0.0
    with P.Context(P.Config(m=10, n=10, rank=2, d=1, precision="fp32")) as ctx:
        ctx.set_matrix(P.TRAIN, [], [], [])
        ctx.set_factors(np.ones((10, 2)), np.ones((10, 2)))
        ctx.epoch(0.1)
        assert ctx.nzsl() == 0.0
        np.testing.assert_array_equal(ctx.get_factors()[0], np.ones((10, 2)))


def test_errors_are_reported_not_crashed():
    with P.Context(P.Config(m=10, n=10, rank=2, d=2)) as ctx:
        with pytest.raises(P.DsgdppError) as e:
            ctx.epoch(0.1)
        assert e.value.status == P.E_STATE
        with pytest.raises(P.DsgdppError) as e:
            ctx.set_matrix(P.TRAIN, [1, 10], [0, 0], [1.0, 2.0])
        assert e.value.status == P.E_INVALID
        with pytest.raises(P.DsgdppError):
            ctx.epoch_explicit(0.1, np.full((4, 2), 9, np.uint32), np.zeros(2, np.uint32))


def _rmse(ctx, ntest):
    return float(np.sqrt(ctx.nzsl(P.TEST) / ntest))


# Test RMSE after 8 constant-step epochs against the sequential FP64 oracle.
# Atomic writes lose no concurrent update and track the oracle to 0.5% (BF16:
# 1%, it rounds every write stochastically); plain stores lose some updates of
# rows updated at the same time, and how many varies run to run (8%).
@pytest.mark.parametrize("precision,write_mode,tol", [
    ("fp64", "atomic", 0.005), ("fp32", "atomic", 0.005), ("bf16", "atomic", 0.01),
    ("fp64", "store", 0.08), ("fp32", "store", 0.08), ("bf16", "store", 0.08)])
@pytest.mark.parametrize("launch", ["stream", "graph"])
def test_hogwild_tracks_fp64_oracle(precision, write_mode, tol, launch):
    p = synth.make(20000, 20000, 400000, 40000, rank_true=10, r=10, noise=0.1, seed=3)
    d = 4
    ref, ctx = _pair(p, 10, d, precision=precision, exec="hogwild", launch=launch,
                     write_mode=write_mode, layout="shuffled")
    with ctx:
        ctx.seed(9)
        ref.seed(9)
        eps = 0.01
        for _ in range(8):
            ctx.epoch(eps)
            ref.epoch(eps)
        got = _rmse(ctx, len(p.tvals))
        want = float(np.sqrt(ref.nzsl(1) / len(p.tvals)))
        start = float(np.sqrt(np.sum((p.tvals - np.einsum("ij,ij->i", p.W0[p.trows],
                                                          p.H0[p.tcols])) ** 2) / len(p.tvals)))
        assert want < 0.9 * start  # the run made progress
        assert abs(got - want) <= tol * want, (got, want)


# Records in runs of one H row (or W row) per group: the run's updates of the
# shared row are sequential and written once; the same tolerances hold.
@pytest.mark.parametrize("layout", ["col_runs", "row_runs"])
@pytest.mark.parametrize("precision,write_mode,tol", [
    ("fp64", "atomic", 0.005), ("fp32", "atomic", 0.005), ("bf16", "atomic", 0.01),
    ("fp32", "store", 0.08)])
def test_hogwild_runs_layout_tracks_fp64_oracle(layout, precision, write_mode, tol):
    p = synth.make(20000, 20000, 400000, 40000, rank_true=10, r=10, noise=0.1, seed=3)
    ref, ctx = _pair(p, 10, 4, precision=precision, exec="hogwild", launch="graph",
                     write_mode=write_mode, layout=layout)
    with ctx:
        ctx.seed(9)
        ref.seed(9)
        for _ in range(8):
            ctx.epoch(0.01)
            ref.epoch(0.01)
        got = _rmse(ctx, len(p.tvals))
        want = float(np.sqrt(ref.nzsl(1) / len(p.tvals)))
        assert abs(got - want) <= tol * want, (got, want)


@pytest.mark.parametrize("layout", ["shuffled", "col_runs", "row_runs"])
def test_hogwild_truncation_bounds_every_factor(layout):
    p = _problem(m=3000, n=2000, nnz=60000, ntest=100, r=12)
    cfg = P.Config(m=p.m, n=p.n, rank=12, d=4, precision="fp32", write_mode="store",
                   truncate=(-0.2, 0.25), layout=layout)
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_factors(np.clip(p.W0, -0.2, 0.25), np.clip(p.H0, -0.2, 0.25))
        for _ in range(3):
            ctx.epoch(0.05)
        W, H = ctx.get_factors()
    assert W.min() >= -0.2 and W.max() <= 0.25 and H.min() >= -0.2 and H.max() <= 0.25


def test_hogwild_lazy_l2_scaling_matches_exact():
    # with no training entries the epoch is pure RegularizeL2 scaling: W is
    # scaled 2d times, each H column block d times
    m, n, r, d = 64, 64, 8, 4
    rng = np.random.default_rng(0)
    W0, H0 = rng.uniform(-1, 1, (m, r)), rng.uniform(-1, 1, (n, r))
    outs = []
    for prec, ex in (("fp64", "replay"), ("fp32", "hogwild"), ("fp64", "hogwild")):
        cfg = P.Config(m=m, n=n, rank=r, d=d, precision=prec, exec=ex, update="Nzsl",
                       regularize="L2", regularize_lambda=0.5, loss="Nzsl")
        with P.Context(cfg) as ctx:
            ctx.set_matrix(P.TRAIN, [], [], [])
            ctx.set_factors(W0, H0)
            sched, seeds = P.draw_schedule(P.Random32(4), d, "COWOR")
            ctx.epoch_explicit(0.3, sched, seeds)
            outs.append(ctx.get_factors())
    for W, H in outs[1:]:
        np.testing.assert_allclose(W, outs[0][0], rtol=2e-6)
        np.testing.assert_allclose(H, outs[0][1], rtol=2e-6)


def test_epoch_time_is_reported():
    p = _problem()
    _, ctx = _pair(p, 10, 2, precision="fp32", exec="hogwild")
    with ctx:
        ctx.epoch(0.01)
        assert ctx.last_epoch_ms() > 0


# One persistent launch per epoch: a block starts when the blocks it depends on
# (its task's previous block, the previous block on its column block) are done.
@pytest.mark.parametrize("precision,tol", [("fp64", 0.005), ("fp32", 0.005), ("bf16", 0.01)])
@pytest.mark.parametrize("sgd_order", ["SEQ", "WOR"])
@pytest.mark.parametrize("layout", ["col_runs", "row_runs"])
def test_persistent_epoch_tracks_fp64_oracle(precision, tol, sgd_order, layout):
    p = synth.make(20000, 20000, 400000, 40000, rank_true=10, r=10, noise=0.1, seed=3)
    ref, ctx = _pair(p, 10, 4, precision=precision, exec="hogwild", launch="persistent",
                     layout=layout, sgd_order=sgd_order)
    with ctx:
        ctx.seed(9)
        ref.seed(9)
        for _ in range(8):
            ctx.epoch(0.01)
            ref.epoch(0.01)
        got = _rmse(ctx, len(p.tvals))
        want = float(np.sqrt(ref.nzsl(1) / len(p.tvals)))
        assert abs(got - want) <= tol * want, (got, want)


def test_persistent_epoch_kernel_timing_and_unsupported_forms():
    p = _problem(m=3000, n=2000, nnz=60000, ntest=100, r=12)
    cfg = P.Config(m=p.m, n=p.n, rank=12, d=8, launch="persistent", layout="col_runs")
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_factors(p.W0, p.H0)
        ctx.set_kernel_timing(True)
        for _ in range(3):
            ctx.epoch(0.01)
        ms, launches = ctx.kernel_timing()
        assert launches == 3 and ms > 0
    for bad in (dict(sgd_order="WR"), dict(write_mode="store"), dict(layout="shuffled"),
                dict(exec="replay", precision="fp64")):
        with pytest.raises(P.DsgdppError):
            P.Context(P.Config(m=p.m, n=p.n, rank=12, d=8, launch="persistent",
                               **dict(dict(layout="col_runs"), **bad)))


def test_persistent_epoch_wait_limit_gives_up_and_the_context_recovers():
    # the bounded dependency wait of the one-launch epoch (in place of the
    # reference's unbounded sub-epoch barrier, mf/sgd/dsgdpp_impl.h:259-263):
    # with a zero limit the first unmet dependency ends the epoch with an error
    # status, and the next epoch on the same context runs normally.  Every
    # sub-epoch here has ~120 chunks against thousands of resident warps, so
    # warps holding later sub-epochs' tickets meet unfinished dependencies.
    p = _problem(m=3000, n=2000, nnz=60000, ntest=600, r=12)
    cfg = P.Config(m=p.m, n=p.n, rank=12, d=8, launch="persistent", layout="col_runs")
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
        ctx.set_factors(p.W0, p.H0)
        ctx.seed(1)
        ctx.epoch(0.01)
        ctx.set_wait_limit(0.0)
        with pytest.raises(P.DsgdppError) as err:
            ctx.epoch(0.01)
        assert err.value.status == P.E_CUDA and "gave up" in str(err.value)
        ctx.set_wait_limit(1.0)
        before = ctx.nzsl(P.TEST)
        for _ in range(3):
            ctx.epoch(0.01)
        after = ctx.nzsl(P.TEST)
        W, H = ctx.get_factors()
        assert np.isfinite(W).all() and np.isfinite(H).all()
        assert after < before
    with pytest.raises(P.DsgdppError):
        with P.Context(cfg) as ctx:
            ctx.set_wait_limit(-1.0)


def test_small_cpu_workload_replay_run_matches_oracle():
    # the reference's CPU-runnable case at full size: 100,000 x 100,000, 1M
    # uniform entries (+100k test), rank 10, FP64, Nzsl_L2(1), d = 4 (4 x 8
    # blocks), BoldDriver(0.001); 3 epochs of the 50 (the oracle is sequential)
    p = synth.make(100_000, 100_000, 1_000_000, 100_000, rank_true=10, r=10, noise=0.1, seed=2024)
    ref, ctx = _pair(p, 10, 4, precision="fp64", exec="replay", launch="graph")
    with ctx:
        ctx.seed(1)
        ref.seed(1)
        tr = ctx.run(3, "BoldDriver", 0.001)
        rt = ref.run(3, "BoldDriver", 0.001)
        for k, row in enumerate(tr):
            assert row["loss"] == pytest.approx(rt[k, 0], rel=LOSS_RTOL)
            assert row["test_loss"] == pytest.approx(rt[k, 1], rel=LOSS_RTOL)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


# ---- DSGD (d x d blocking, d sub-epochs; mf/sgd/dsgd_impl.h) -------------------
@pytest.mark.parametrize("stratum_order", ["SEQ", "RSEQ", "WR", "WOR", "COWOR"])
@pytest.mark.parametrize("sgd_order", ["SEQ", "WOR"])
def test_dsgd_replay_master_rng_epochs_bit_exact(stratum_order, sgd_order):
    p = _problem()
    d = 3
    ref = O.Problem(p.m, p.n, 10, d, p.rows, p.cols, p.vals, p.trows, p.tcols, p.tvals,
                    method="dsgd")
    ref.configure(sgd_order=sgd_order, stratum_order=stratum_order, update_lambda=0.5)
    ref.set_factors(p.W0, p.H0)
    cfg = P.Config(m=p.m, n=p.n, rank=10, d=d, precision="fp64", exec="replay", method="dsgd",
                   sgd_order=sgd_order, stratum_order=stratum_order, update_lambda=0.5)
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
        ctx.set_factors(p.W0, p.H0)
        assert ctx.block_nnz(P.TRAIN).shape == (d, d)
        np.testing.assert_array_equal(ctx.block_nnz(P.TRAIN), ref.block_nnz(0))
        ctx.seed(5)
        ref.seed(5)
        for _ in range(3):
            ctx.epoch(0.02)
            ref.epoch(0.02)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)
        assert ctx.loss() == pytest.approx(ref.loss(), rel=LOSS_RTOL)


def test_dsgd_replay_l2_regularize_and_run_trace():
    p = _problem(m=800, n=600, nnz=10000, ntest=1000)
    ref = O.Problem(p.m, p.n, 10, 4, p.rows, p.cols, p.vals, p.trows, p.tcols, p.tvals,
                    method="dsgd")
    ref.configure(regularize="L2", regularize_lambda=0.05)
    ref.set_factors(p.W0, p.H0)
    cfg = P.Config(m=p.m, n=p.n, rank=10, d=4, precision="fp64", exec="replay", method="dsgd",
                   regularize="L2", regularize_lambda=0.05)
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
        ctx.set_factors(p.W0, p.H0)
        ctx.seed(42)
        ref.seed(42)
        tr = ctx.run(5, "BoldDriver", 0.01)
        rt = ref.run(5, "BoldDriver", 0.01)
        for k, row in enumerate(tr):
            assert row["loss"] == pytest.approx(rt[k, 0], rel=LOSS_RTOL)
            assert row["test_loss"] == pytest.approx(rt[k, 1], rel=LOSS_RTOL)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


@pytest.mark.parametrize("precision,tol", [("fp32", 0.005), ("bf16", 0.01)])
@pytest.mark.parametrize("launch", ["graph", "persistent"])
def test_dsgd_hogwild_tracks_fp64_oracle(precision, tol, launch):
    p = synth.make(20000, 20000, 400000, 40000, rank_true=10, r=10, noise=0.1, seed=3)
    ref = O.Problem(p.m, p.n, 10, 4, p.rows, p.cols, p.vals, p.trows, p.tcols, p.tvals,
                    method="dsgd")
    ref.configure(regularize="L2", regularize_lambda=0.02)
    ref.set_factors(p.W0, p.H0)
    cfg = P.Config(m=p.m, n=p.n, rank=10, d=4, precision=precision, launch=launch,
                   method="dsgd", regularize="L2", regularize_lambda=0.02)
    with P.Context(cfg) as ctx:
        ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
        ctx.set_matrix(P.TEST, p.trows, p.tcols, p.tvals)
        ctx.set_factors(p.W0, p.H0)
        ctx.seed(9)
        ref.seed(9)
        for _ in range(8):
            ctx.epoch(0.01)
            ref.epoch(0.01)
        got = _rmse(ctx, len(p.tvals))
        want = float(np.sqrt(ref.nzsl(1) / len(p.tvals)))
        assert abs(got - want) <= tol * want, (got, want)


def test_dsgd_blocking_limits_and_batch_rejection():
    p = _problem(m=50, n=5, nnz=100, ntest=10)
    P.Context(P.Config(m=p.m, n=p.n, rank=4, d=5, method="dsgd")).close()  # n >= d suffices
    with pytest.raises(P.DsgdppError):
        P.Context(P.Config(m=p.m, n=p.n, rank=4, d=5))  # DSGD++ needs n >= 2d
    prob = dict(m=p.m, n=p.n, rank=4, rows=p.rows, cols=p.cols, vals=p.vals, W=p.W0[:, :4],
                H=p.H0[:, :4])
    with pytest.raises(P.DsgdppError):
        P.Batch(P.Config(m=1, n=1, rank=1, d=1, method="dsgd"), [prob])


# ---- blocked input and caller-held counts (the runner's own data form) ---------------
def _oracle_blocks(ref, d, nb2, which=0):
    parts = [ref.block_records(b1, b2, which) for b1 in range(d) for b2 in range(nb2)]
    bn = np.array([len(x) for _, _, x in parts], np.uint64)
    cat = lambda k: np.concatenate([p[k] for p in parts]) if len(parts) else np.empty(0)
    return bn, cat(0), cat(1), cat(2)


@pytest.mark.parametrize("method", ["dsgdpp", "dsgd"])
def test_set_blocks_matches_set_matrix_and_oracle(method):
    p = _problem()
    d = 3
    nb2 = d if method == "dsgd" else 2 * d
    ref = O.Problem(p.m, p.n, 10, d, p.rows, p.cols, p.vals, p.trows, p.tcols, p.tvals,
                    method=method)
    ref.configure(update_lambda=0.5)
    ref.set_factors(p.W0, p.H0)
    cfg = P.Config(m=p.m, n=p.n, rank=10, d=d, precision="fp64", exec="replay", method=method,
                   update_lambda=0.5)
    bn, li, lj, lx = _oracle_blocks(ref, d, nb2)
    tbn, ti, tj, tx = _oracle_blocks(ref, d, nb2, which=1)
    with P.Context(cfg) as ctx:
        ctx.set_blocks(P.TRAIN, bn, li, lj, lx)
        ctx.set_blocks(P.TEST, tbn, ti, tj, tx)
        ctx.set_factors(p.W0, p.H0)
        np.testing.assert_array_equal(ctx.block_nnz(P.TRAIN).ravel(), bn)
        a1, a2, _ = ctx.nnz12()
        r1, r2, _ = ref.nnz12()
        np.testing.assert_array_equal(a1, r1)
        np.testing.assert_array_equal(a2, r2)
        ctx.seed(11)
        ref.seed(11)
        for _ in range(2):
            ctx.epoch(0.02)
            ref.epoch(0.02)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)
        assert ctx.nzsl(P.TEST) == pytest.approx(ref.nzsl(1), rel=LOSS_RTOL)


def test_set_blocks_rejects_entries_outside_their_block():
    p = _problem(m=60, n=40, nnz=300, ntest=30)
    d = 2
    cfg = P.Config(m=p.m, n=p.n, rank=4, d=d)
    bn = np.zeros(d * 2 * d, np.uint64)
    bn[0] = 2
    with P.Context(cfg) as ctx:
        # block (0, 0) spans rows [0, 30) and columns [0, 10)
        with pytest.raises(P.DsgdppError, match="outside their block"):
            ctx.set_blocks(P.TRAIN, bn, [0, 30], [0, 1], [1.0, 2.0])
        with pytest.raises(P.DsgdppError, match="outside their block"):
            ctx.set_blocks(P.TRAIN, bn, [0, 1], [0, 10], [1.0, 2.0])
        ctx.set_blocks(P.TRAIN, bn, [0, 29], [0, 9], [1.0, 2.0])
        assert int(ctx.block_nnz(P.TRAIN).sum()) == 2


def test_set_counts_replaces_the_update_weights():
    p = _problem()
    cfg = dict(m=p.m, n=p.n, rank=10, d=3, precision="fp64", exec="replay")
    with P.Context(P.Config(**cfg)) as a, P.Context(P.Config(**cfg)) as b:
        for ctx in (a, b):
            ctx.set_matrix(P.TRAIN, p.rows, p.cols, p.vals)
            ctx.set_factors(p.W0, p.H0)
            ctx.seed(4)
        n1, n2, _ = a.nnz12()
        b.set_counts(n1, n2)  # the same counts: the same run, bit for bit
        a.epoch(0.02)
        b.epoch(0.02)
        np.testing.assert_array_equal(a.get_factors()[0], b.get_factors()[0])
        b.set_counts(n1 * 2, n2 * 2)  # doubled counts halve the regularization weights
        a.epoch(0.02)
        b.epoch(0.02)
        assert not np.array_equal(a.get_factors()[0], b.get_factors()[0])
        m1, m2, _ = b.nnz12()
        np.testing.assert_array_equal(m1, n1 * 2)
        with pytest.raises(P.DsgdppError):
            b.set_counts(np.full(p.m, 1 << 33, np.uint64), n2)


@pytest.mark.parametrize("r,m,n,nnz,d,kind", [
    (10, 4000, 3000, 60000, 1, "uniform"),   # one task, more than 2^11 rounds' worth of places
    (16, 300, 200, 9000, 2, "uniform"),      # rows and columns repeat within what is in hand
    (17, 90, 2, 150, 1, "uniform"),          # two columns: nearly every record waits for another
    (5, 64, 4000, 30000, 1, "zipf"),         # hot rows and columns: long chains
    (65, 500, 400, 5000, 3, "zipf"),
    (200, 300, 200, 3000, 2, "zipf"),
    (256, 40, 8, 200, 4, "uniform")])        # blocks of a few entries, the widest rows
def test_replay_runs_independent_records_together_bit_exact(r, m, n, nnz, d, kind):
    p = _problem(m=m, n=n, nnz=nnz, ntest=10, r=r, kind=kind)
    ref, ctx = _pair(p, r, d, regularize="L2", regularize_lambda=0.05)
    with ctx:
        R = P.Random32(r)
        for _ in range(2):
            sched, seeds = P.draw_schedule(R, d, "COWOR")
            ctx.epoch_explicit(0.01, sched, seeds)
            ref.epoch_explicit(0.01, sched, seeds)
        W, H = ctx.get_factors()
        Wr, Hr = ref.get_factors()
        np.testing.assert_array_equal(W, Wr)
        np.testing.assert_array_equal(H, Hr)


def test_replay_of_one_column_outlasts_the_round_numbers():
    # nearly every record lies in one column, so a round runs one or two of
    # them and the round numbers (2^11) start over
    rng = np.random.default_rng(3)
    rows = np.concatenate([np.arange(6000), rng.permutation(6000)[:50]]).astype(np.uint32)
    cols = np.concatenate([np.zeros(6000), np.ones(50)]).astype(np.uint32)
    vals = rng.standard_normal(6050)
    W0, H0 = rng.uniform(-.5, .5, (6000, 7)), rng.uniform(-.5, .5, (2, 7))
    ref = O.Problem(6000, 2, 7, 1, rows, cols, vals, rows[:5], cols[:5], vals[:5])
    ref.configure()
    ref.set_factors(W0, H0)
    with P.Context(P.Config(m=6000, n=2, rank=7, d=1, precision="fp64", exec="replay",
                            launch="stream")) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        sched, seeds = P.draw_schedule(P.Random32(5), 1, "WOR")
        ctx.epoch_explicit(0.001, sched, seeds)
        ref.epoch_explicit(0.001, sched, seeds)
        for a, b in zip(ctx.get_factors(), ref.get_factors()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision,r", [
    ("fp32", 3), ("fp32", 8), ("fp32", 16), ("fp32", 24), ("fp32", 28), ("fp32", 64),
    ("fp32", 90), ("fp32", 96), ("fp32", 132), ("fp32", 136), ("fp32", 260), ("fp32", 508),
    ("fp32", 512), ("bf16", 8), ("bf16", 16), ("bf16", 20), ("bf16", 40), ("bf16", 192),
    ("bf16", 264), ("bf16", 512), ("bf16", 1016), ("bf16", 1024), ("fp64", 5), ("fp64", 256)])
@pytest.mark.parametrize("nnz", [1, 31, 4129])
def test_losses_and_norms_of_every_row_mapping(precision, r, nnz):
    # against FP64 sums over the stored factors; the sums have at most 4129 r
    # terms of one sign, so any order of adding them agrees to 1e-12
    m, n = 70, 61
    rng = np.random.default_rng(r + nnz)
    keys = rng.permutation(m * n)[:nnz]
    rows, cols = (keys // n).astype(np.uint32), (keys % n).astype(np.uint32)
    vals = rng.standard_normal(nnz)
    W0, H0 = rng.uniform(-.5, .5, (m, r)), rng.uniform(-.5, .5, (n, r))
    lanes = 32 if precision == "fp32" and r > 128 else 0  # the epoch kernels' own mapping
    with P.Context(P.Config(m=m, n=n, rank=r, d=2, precision=precision,
                            lanes_per_nnz=lanes)) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        W, H = ctx.get_factors()
        x = vals if precision == "fp64" else vals.astype(np.float32).astype(np.float64)
        want = float(np.sum((x - np.einsum("ij,ij->i", W[rows], H[cols])) ** 2))
        w2, h2 = np.sum(W * W, 1), np.sum(H * H, 1)
        c1, c2 = np.bincount(rows, minlength=m), np.bincount(cols, minlength=n)
        near = dict(rtol=LOSS_RTOL, atol=0)
        np.testing.assert_allclose(ctx.nzsl(P.TRAIN), want, **near)
        np.testing.assert_allclose(ctx.l2(), (w2.sum(), h2.sum()), **near)
        np.testing.assert_allclose(ctx.nzl2(), (c1 @ w2, c2 @ h2), **near)
        np.testing.assert_allclose(ctx.loss(), want + w2.sum() + h2.sum(), **near)
        ctx.save_factors()
        ctx.set_factors(W0 * 1.5, H0)
        moved = np.sqrt(np.sum((ctx.get_factors()[0] - W) ** 2, 1))
        np.testing.assert_allclose(ctx.update_norms(), (moved.sum() / (m + n), moved.max()), **near)


@pytest.mark.parametrize("m,n,r", [(26214, 26215, 10), (131072, 3, 2), (131073, 200, 2),
                                   (400001, 300007, 3), (1000, 900, 700)])
def test_factors_through_pageable_and_page_locked_arrays(m, n, r):
    # 2 MiB - 32 bytes (copied as they are), exactly 2 MiB, a byte count just
    # above, and many pieces with an odd end
    import torch
    rng = np.random.default_rng(m)
    W0, H0 = rng.standard_normal((m, r)), rng.standard_normal((n, r))
    lanes = 32 if r > 256 else 0
    with P.Context(P.Config(m=m, n=n, rank=min(r, 256), d=1, precision="fp64",
                            lanes_per_nnz=lanes)) as ctx:
        W0, H0 = W0[:, :256].copy(), H0[:, :256].copy()
        for lock in (False, True):
            give = (lambda a: torch.from_numpy(a).pin_memory().numpy()) if lock else np.copy
            ctx.set_factors(give(W0), give(H0))
            W, H = ctx.get_factors()
            np.testing.assert_array_equal(W, W0)
            np.testing.assert_array_equal(H, H0)
            W, H = give(np.zeros_like(W0)), give(np.zeros_like(H0))
            ctx.get_factors_into(W, H)
            np.testing.assert_array_equal(W, W0)
            np.testing.assert_array_equal(H, H0)


@pytest.mark.parametrize("nnz", [200_000, 262_144, 524_289, 1_300_001])
def test_matrix_from_pageable_and_page_locked_arrays(nnz):
    import torch
    rng = np.random.default_rng(nnz)
    rows = rng.integers(0, 5000, nnz).astype(np.uint32)  # some pairs repeat: values are summed
    cols = rng.integers(0, 4000, nnz).astype(np.uint32)
    vals = rng.standard_normal(nnz)
    lock = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a
                                      ).pin_memory().numpy().view(a.dtype)
    got = []
    for give in (np.copy, lock):
        with P.Context(P.Config(m=5000, n=4000, rank=4, d=3, precision="fp64")) as ctx:
            ctx.set_matrix(P.TRAIN, give(rows), give(cols), give(vals))
            ctx.set_factors(np.zeros((5000, 4)), np.zeros((4000, 4)))
            got.append((ctx.block_nnz(), *ctx.nnz12()[:2], ctx.nzsl(P.TRAIN)))
            bad = rows.copy()
            bad[nnz // 2] = 5000  # refused while the values are still on their way
            with pytest.raises(P.DsgdppError):
                ctx.set_matrix(P.TRAIN, give(bad), give(cols), give(vals))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("r", [3, 10, 50, 130])
def test_losses_of_infinite_factors_leave_out_the_rows_padding(r):
    # an infinite step times the padding's zeros is NaN; the loss of the
    # factors themselves is infinite
    with P.Context(P.Config(m=4, n=4, rank=r, d=1, precision="fp32", update="Nzsl", loss="Nzsl",
                            lanes_per_nnz=32 if r > 128 else 0)) as ctx:
        at = np.zeros(1, np.uint32)
        ctx.set_matrix(P.TRAIN, at, at, np.ones(1))
        ctx.set_matrix(P.TEST, at, at, np.ones(1))
        ctx.set_factors(np.full((4, r), 1e20), np.full((4, r), 1e20))
        ctx.seed(1)
        ctx.epoch(0.01)
        W, H = ctx.get_factors()
        assert (1.0 - W[0] @ H[0]) ** 2 == np.inf
        assert ctx.loss() == np.inf and ctx.nzsl(P.TEST) == np.inf


@pytest.mark.parametrize("r", [2, 7, 10, 33, 64, 255])
def test_fp64_nonzero_weighted_loss_forms_each_row_as_the_reference(r):
    # one row of each factor is not zero, so the sum over the rows is exact
    rng = np.random.default_rng(r)
    m, n = 50, 40
    keys = rng.permutation(m * n)[:900]
    rows, cols = (keys // n).astype(np.uint32), (keys % n).astype(np.uint32)
    with P.Context(P.Config(m=m, n=n, rank=r, d=2, precision="fp64")) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, rng.standard_normal(900))
        for i, j in ((0, 0), (17, 23), (m - 1, n - 1)):
            W, H = np.zeros((m, r)), np.zeros((n, r))
            W[i], H[j] = rng.standard_normal(r), rng.standard_normal(r)
            ctx.set_factors(W, H)
            want = []
            for x, count in ((W[i], np.sum(rows == i)), (H[j], np.sum(cols == j))):
                total = 0.0
                for z in range(r):
                    total += float(x[z]) * float(x[z])
                want.append(float(count) * total)
            assert ctx.nzl2() == tuple(want)


@pytest.mark.parametrize("launch", ["graph", "stream"])
@pytest.mark.parametrize("regularize", ["None", "L2"])
def test_sub_epochs_without_entries_keep_the_others_in_order(launch, regularize):
    # column blocks 2 and 3 are empty, so sub-epochs 1 and 3 are; 0 and 2 update
    # the same rows, each row and column once, so their order is the result
    M, r = 40_000, 16
    rng = np.random.default_rng(5)
    rows = np.concatenate([np.arange(2 * M), np.arange(2 * M)]).astype(np.uint32)
    # the first half of the rows is in block 0 and then 1, the second in 1 and then 0
    cols = np.concatenate([rng.permutation(M), M + rng.permutation(M), M + rng.permutation(M),
                           rng.permutation(M)]).astype(np.uint32)
    vals = rng.standard_normal(4 * M)
    W0, H0 = rng.uniform(-.5, .5, (2 * M, r)), rng.uniform(-.5, .5, (4 * M, r))
    kw = dict(regularize=regularize, regularize_lambda=0.05 if regularize == "L2" else 0.0)
    ref = O.Problem(2 * M, 4 * M, r, 2, rows, cols, vals, rows[:5], cols[:5], vals[:5])
    ref.configure(**kw)
    ref.set_factors(W0, H0)
    with P.Context(P.Config(m=2 * M, n=4 * M, rank=r, d=2, precision="fp64", exec="hogwild",
                            launch=launch, **kw)) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        sched = np.array([0, 1, 2, 3, 1, 0, 3, 2], np.uint32)
        for _ in range(3):
            ctx.epoch_explicit(0.05, sched, [1, 2])
            ref.epoch_explicit(0.05, sched, [1, 2])
        for a, b in zip(ctx.get_factors(), ref.get_factors()):
            # L2: twelve scales held in FP32, each off by up to 6e-8 of its value
            np.testing.assert_allclose(a, b, rtol=0, atol=5e-6 if regularize == "L2" else 1e-12)


@pytest.mark.parametrize("r", [1, 2, 3, 8, 9])
@pytest.mark.parametrize("kind", ["uniform", "zipf"])
def test_replay_of_few_elements_per_lane_bit_exact(r, kind):
    p = _problem(m=300, n=250, nnz=12000, ntest=10, r=r, kind=kind)
    ref, ctx = _pair(p, r, 2, regularize="L2", regularize_lambda=0.05)
    with ctx:
        R = P.Random32(r)
        for _ in range(2):
            sched, seeds = P.draw_schedule(R, 2, "COWOR")
            ctx.epoch_explicit(0.01, sched, seeds)
            ref.epoch_explicit(0.01, sched, seeds)
        for a, b in zip(ctx.get_factors(), ref.get_factors()):
            np.testing.assert_array_equal(a, b)


def test_replay_of_a_block_whose_places_count_from_a_new_base():
    # a round hands out at most 128 records, so the round numbers (2^11) start
    # over at least once between places 2^19 and 2^19 + 2^18, with all places
    # after that counted from a base above 0
    m, n, nnz, r = 3000, 2500, 900_000, 4
    rng = np.random.default_rng(11)
    keys = rng.permutation(m * n)[:nnz]
    rows, cols = (keys // n).astype(np.uint32), (keys % n).astype(np.uint32)
    vals = rng.standard_normal(nnz)
    W0, H0 = rng.uniform(-.5, .5, (m, r)), rng.uniform(-.5, .5, (n, r))
    ref = O.Problem(m, n, r, 1, rows, cols, vals, rows[:5], cols[:5], vals[:5],
                    method="dsgd")  # one block
    ref.configure()
    ref.set_factors(W0, H0)
    with P.Context(P.Config(m=m, n=n, rank=r, d=1, precision="fp64", exec="replay",
                            launch="stream", method="dsgd")) as ctx:
        ctx.set_matrix(P.TRAIN, rows, cols, vals)
        ctx.set_factors(W0, H0)
        ctx.epoch_explicit(0.001, [0], [5])
        ref.epoch_explicit(0.001, [0], [5])
        for a, b in zip(ctx.get_factors(), ref.get_factors()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("r", [1, 10, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("d,nnz", [(1, 1), (1, 40), (20, 900), (160, 6000)])
@pytest.mark.parametrize("update,truncate", [("Nzsl", None), ("Nzsl_L2", None),
                                             ("Nzsl_Nzl2", (-0.4, 0.4))])
def test_replay_of_blocks_of_few_records_bit_exact(r, d, nnz, update, truncate):
    # from one record to some ten a block, walked or run in rounds by the rank
    p = _problem(m=500, n=400, nnz=nnz, ntest=10, r=r)
    ref, ctx = _pair(p, r, d, update=update, update_lambda=0.5, truncate=truncate)
    with ctx:
        R = P.Random32(r)
        for _ in range(2):
            sched, seeds = P.draw_schedule(R, d, "COWOR")
            ctx.epoch_explicit(0.02, sched, seeds)
            ref.epoch_explicit(0.02, sched, seeds)
        for a, b in zip(ctx.get_factors(), ref.get_factors()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("r", [133, 245, 260, 500, 515, 773, 270, 510, 700, 1023])
def test_losses_of_bf16_ranks_that_end_inside_a_vector_of_eight_lanes_and_more(r):
    test_losses_and_norms_of_every_row_mapping("bf16", r, 4129)
