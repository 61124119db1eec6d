"""Which kernel a plan, a handle and a batch run, and that a schedule which is set, tuned or reported is
one of the kernel that it says."""
import numpy as np
import pytest

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300 import batch, gen

pytestmark = pytest.mark.gpu


def _plan(vt, a, *cfg):
    import torch
    return sp.Plan(vt, a.m, a.n, torch.from_numpy(a.row_ptr).cuda(), torch.from_numpy(a.col).cuda(),
                   None, *cfg)


def _handle(vt, a, cfg=None):
    h = sp.BhsparseSpmvCuda(vt)
    if cfg is not None:
        assert h.set_config(*cfg) == 0, h.last_error
    dt = sp.host_dtype(vt)
    y = np.zeros(a.m, dt)
    assert h.prepare_mem(a.m, a.n, a.nnz, a.row_ptr, a.col, a.val.astype(dt), np.ones(a.n, dt), y) == 0
    return h, y


@pytest.mark.parametrize("vt", [sp.VALUE_F64, sp.VALUE_F32, sp.VALUE_MIXED_F32, sp.VALUE_MIXED_BF16])
def test_plan_and_handle_report_their_kernel(cuda_ok, capfd, monkeypatch, vt):
    monkeypatch.setenv("BHSP_LOG_SCHEDULE", "1")
    for a, kernel in ((gen.stencil3d(30, 30, 30), (1, 28)), (gen.stencil2d(90, 80), (1, 8)),
                      (gen.powerlaw(20_000, seed=3), (0, 0))):
        p = _plan(vt, a)
        assert p.kernel() == kernel and p.launches == (1 if kernel[0] else 2)
        if kernel[0]:
            p.set_grid(False)
            assert p.kernel() == (0, 0)
            p.set_grid(None)
            assert p.kernel() == kernel
            p.set_variant(l2_only=p.gather_path()[2])
            assert p.kernel() == (0, 0)
        p.close()
        capfd.readouterr()
        h, _ = _handle(vt, a)
        assert h.kernel() == kernel
        assert ("row kernel" in capfd.readouterr().err) == (kernel[0] > 0)
        h.close()


@pytest.mark.parametrize("k", [1, 2, 4, 8])
def test_batch_reports_its_lists(cuda_ok, k):
    regular, power = gen.stencil3d(40, 40, 40), gen.powerlaw(20_000, seed=3)
    wide = gen.blockdiag(4096, 4096, 512)
    for mats, lists, tiles, variant in (([regular] * 2, True, False, (False, False)),
                                        ([regular, power], True, True, (False, True)),
                                        ([regular, wide], True, True, (k == 1, False)),
                                        ([power], False, False, (False, False))):
        b = batch.Batch(mats, k=k)
        info = b.info()
        assert (info["row_lists"] > 0) == lists and (info["tile_workers"] > 0) == tiles
        assert (info["workers_one_head"], info["workers_x_l2_only"]) == variant
        b.set_variant(l2_only=info["x_l2_only"])
        info = b.info()
        assert info["row_lists"] == info["tile_workers"] == 0 and info["launches"] == 2
        b.close()


@pytest.mark.parametrize("vt", [sp.VALUE_F64, sp.VALUE_F32, sp.VALUE_MIXED_F32, sp.VALUE_MIXED_BF16])
@pytest.mark.parametrize("cfg", [(8, 4, 4, 0), (16, 2, 4, 2), (0, 0, 0, -1)])
def test_a_schedule_that_the_caller_sets_runs(cuda_ok, vt, cfg):
    """bhsp_set_config: the handle runs the tile kernel, also on a matrix that takes the row kernel
    without it, and y is the exact sum."""
    a = gen.stencil3d(30, 20, 25)
    a.val = gen.uniform_int(a.nnz, 8, 10) - 4.0
    want = np.bincount(np.repeat(np.arange(a.m), np.diff(a.row_ptr)), a.val, a.m)
    for c, rows in ((None, True), (cfg, False)):
        h, y = _handle(vt, a, c)
        assert (h.kernel()[0] > 0) == rows
        assert h.run_benchmark() == 0 and h.get_y() == 0
        assert (y == want).all()
        h.close()


def _tune_args(a):
    import torch
    return (torch.from_numpy(a.row_ptr).cuda(), torch.from_numpy(a.col).cuda(),
            torch.from_numpy(a.val).cuda().float(), torch.rand(a.n, device="cuda"),
            torch.empty(a.m, device="cuda"))


def test_autotune_times_the_tile_kernel_also_for_row_matrices(cuda_ok, tmp_path):
    """Two matrices with the same row lengths and one cache: random columns (the row kernel) and near
    ones (the tile kernel).  The table that the first leaves for the second is of the tile kernel: its
    slowest candidate takes at least 1.3 times its fastest (1.47 is the least of the 1241 matrices of
    4 M non-zeros and more in the tuner's FP32 dataset; one kernel timed 32 times differs by a few
    per cent)."""
    from benchmark_spmv_using_csr_gb300 import tune
    rng = np.random.default_rng(4)
    lens = rng.integers(0, 28, 400_000)
    spread = gen.from_row_lengths(lens, lens.size, seed=5)
    row = np.repeat(np.arange(lens.size), lens)
    near = gen.CSR(spread.m, spread.n, spread.row_ptr,
                   ((row + np.arange(row.size) - spread.row_ptr[row]) % lens.size).astype(np.int32),
                   spread.val)
    kernels = []
    for a in (spread, near):
        p = _plan(sp.VALUE_F32, a)
        kernels.append(p.kernel()[0] > 0)
        p.close()
    assert kernels == [True, False]
    cache = tune.TuneCache(str(tmp_path / "cache.json"))
    ms, best = cache.tune(sp.VALUE_F32, *_tune_args(spread), warmup=1, reps=3)
    got, got_best = cache.tune(sp.VALUE_F32, *_tune_args(near))
    assert got_best == best and np.array_equal(got, ms)  # from the cache
    ms = ms[np.isfinite(ms)]
    assert ms.max() >= 1.3 * ms.min(), (ms.min(), ms.max())


def test_no_sweep_for_a_row_matrix(cuda_ok, tmp_path):
    """With the network's threshold above any probability every matrix takes the sweep, except one
    whose plan runs the row kernel: it keeps the network's pick."""
    import os

    from benchmark_spmv_using_csr_gb300 import mlp, tune
    net = os.path.join(os.path.dirname(sp.__file__), "tuner_data", "gb300_f32_tuner.bin")
    d = mlp.read_network(net)
    path = str(tmp_path / "net.bin")
    mlp.write_network(path, d["value_type"], d["hidden"], 2.0, d["mean"], d["std"], d["candidates"],
                      d["params"], d["risk"])
    for a, source in ((gen.powerlaw(50_000, seed=6), sp.SCHEDULE_SWEEP),
                      (gen.stencil3d(40, 40, 40), sp.SCHEDULE_LEARNED)):
        args = _tune_args(a)
        got = tune.choose_schedule(sp.VALUE_F32, *args, tuner=path)
        assert got["source"] == source and got["config"] in tune.candidates()
        p = sp.Plan(sp.VALUE_F32, a.m, a.n, args[0], args[1], None, *got["config"])
        assert (p.kernel()[0] > 0) == (source == sp.SCHEDULE_LEARNED)
        p.close()
