"""The work that users of the library have it do, as cases that a timing harness runs.

Three ways in, each as a program calls it:

* ``plan``: y = A.x on device buffers the program owns.  The schedule comes from
  ``tune.choose_schedule`` and is fixed in a ``Plan`` once per matrix; a pass is one
  ``Plan.execute`` (a solver's iteration).
* ``batch``: many matrices of uneven size with 1 to 8 right-hand sides, in a ``Batch`` built once;
  a pass is one ``Batch.execute`` (a graph replay).
* ``handle``: the drop-in class on host arrays.  ``prepare_mem`` once per matrix; a pass is
  ``set_x``, ``run_benchmark`` and ``get_y`` on ordinary (pageable) numpy arrays.

Matrices are the library's own workloads: 5-point and 27-point stencils, power-law rows, uniform
density, block-diagonal dense blocks, one fully dense row, and 90 % empty rows.  A matrix's row
lengths are the quantiles of its distribution in a seeded order, so that the number of
non-zeros follows from the case alone; columns, values and x come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300 import tune
from benchmark_spmv_using_csr_gb300.batch import Batch

VALUE_TYPES = {"f64": sp.VALUE_F64, "f32": sp.VALUE_F32, "mixed_f32": sp.VALUE_MIXED_F32,
               "mixed_bf16": sp.VALUE_MIXED_BF16}
STORE = {"f64": torch.float64, "f32": torch.float32, "mixed_f32": torch.float32,
         "mixed_bf16": torch.bfloat16}
BATCH_KINDS = ("stencil2d", "stencil3d", "powerlaw", "density", "blockdiag")
BLOCK = 32            # block-diagonal: dense blocks of 32 x 32
MAX_LEN = 200_000     # power-law rows are clipped to this
POISSON_MEAN = 8.0    # mean length of the ordinary rows beside a dense row or among empty ones


def listed():
    return [
        # the 2D Laplacian of a small implicit solver: launch latency and the host path
        {"name": "lap2d_256_f64", "use": "plan", "kind": "stencil2d", "nx": 256, "ny": 256,
         "vt": "f64"},
        # the smallest ordinary call: a graph of a few thousand vertices
        {"name": "powerlaw_5k_f32", "use": "plan", "kind": "powerlaw", "m": 5_003, "n": 5_003,
         "vt": "f32"},
        # a large irregular graph, FP64: random gathers from an L2-resident x
        {"name": "powerlaw_4m_f64", "use": "plan", "kind": "powerlaw", "m": 4_194_304,
         "n": 4_194_304, "vt": "f64"},
        # a medium rectangular graph matrix, FP32 storage with compensated sums
        {"name": "powerlaw_700k_mixed_f32", "use": "plan", "kind": "powerlaw", "m": 700_001,
         "n": 900_007, "vt": "mixed_f32"},
        # the large 3D stencil, plain FP64: streaming at the memory's and the FP64 pipe's rate
        {"name": "stencil27_160_f64", "use": "plan", "kind": "stencil3d", "nx": 160, "ny": 160,
         "nz": 160, "vt": "f64"},
        # the same stencil in FP32 storage with compensated sums
        {"name": "stencil27_160_mixed_f32", "use": "plan", "kind": "stencil3d", "nx": 160,
         "ny": 160, "nz": 160, "vt": "mixed_f32"},
        # an odd-sized 3D grid in BF16 storage
        {"name": "stencil27_odd_mixed_bf16", "use": "plan", "kind": "stencil3d", "nx": 121,
         "ny": 97, "nz": 143, "vt": "mixed_bf16"},
        # Poisson rows at uniform density, rectangular, plain FP32
        {"name": "density_300k_f32", "use": "plan", "kind": "density", "m": 300_007,
         "n": 200_003, "vt": "f32"},
        # one constraint that touches every unknown, beside ordinary short rows
        {"name": "dense_row_1m_f64", "use": "plan", "kind": "dense_row", "m": 1_000_003,
         "n": 1_000_003, "vt": "f64"},
        # a batch of independent systems, one right-hand side each
        {"name": "batch_128_k1", "use": "batch", "count": 128, "k": 1},
        # the same kind of batch with eight right-hand sides
        {"name": "batch_64_k8", "use": "batch", "count": 64, "k": 8},
        # the drop-in class driven call by call from host arrays
        {"name": "handle_stencil27_80_f64", "use": "handle", "kind": "stencil3d", "nx": 80,
         "ny": 80, "nz": 80, "vt": "f64"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    use = rng.choices(["plan", "batch", "handle"], [8, 3, 1])[0]
    if use == "batch":
        k = rng.choice([1, 2, 4, 8])
        return {"use": "batch", "count": _log_uniform(rng, 4, 128 if k <= 2 else 64), "k": k}
    if use == "plan":
        vt = rng.choice(["f64", "f32", "mixed_f32", "mixed_bf16"])
        top = 4_000_000
    else:
        vt = rng.choice(["f64", "f32"])
        top = 500_000
    kind = rng.choice(["stencil2d", "stencil3d", "powerlaw", "density", "blockdiag", "dense_row",
                       "empty_rows"])
    c = {"use": use, "kind": kind, "vt": vt}
    m = _log_uniform(rng, 1_000, min(top, 1_000_000) if kind == "density" else top)
    if kind == "stencil2d":
        c["nx"] = max(1, int(m ** 0.5 * rng.uniform(0.6, 1.6)))
        c["ny"] = max(1, m // c["nx"])
    elif kind == "stencil3d":
        c["nx"] = max(1, int(m ** (1 / 3) * rng.uniform(0.7, 1.4)))
        c["ny"] = max(1, int((m / c["nx"]) ** 0.5 * rng.uniform(0.7, 1.4)))
        c["nz"] = max(1, m // (c["nx"] * c["ny"]))
    else:
        c["m"] = m
        c["n"] = m if kind == "blockdiag" or rng.random() < 0.5 else int(m * rng.uniform(0.5, 2)) + 1
    return c


# --- sizes: what follows from the case alone ------------------------------------------------
def _rows_cols(c):
    if c["kind"] == "stencil2d":
        m = c["nx"] * c["ny"]
        return m, m
    if c["kind"] == "stencil3d":
        m = c["nx"] * c["ny"] * c["nz"]
        return m, m
    return c["m"], c["n"]


def _poisson_quantiles(mean, count):
    top = int(mean + 12 * math.sqrt(mean) + 20)
    pmf = [math.exp(-mean)]
    for i in range(1, top):
        pmf.append(pmf[-1] * mean / i)
    u = (np.arange(count) + 0.5) / count
    return np.searchsorted(np.cumsum(pmf), u).astype(np.int64)


@functools.lru_cache(maxsize=64)
def _lengths(kind, m, n):
    """Row lengths of a matrix without a grid, as quantiles in ascending order of the quantile."""
    if kind == "powerlaw":  # a Zipf(2.1) tail, 5 % of the rows empty
        empty = int(0.05 * m)
        u = (np.arange(m - empty) + 0.5) / max(1, m - empty)
        ln = np.floor(1.98 * u ** (-1 / 1.1)).astype(np.int64)
        return np.concatenate([np.zeros(empty, np.int64), np.clip(ln, 1, min(MAX_LEN, n))])
    if kind == "density":  # uniform density 1e-4
        return np.minimum(_poisson_quantiles(1e-4 * n, m), n)
    if kind == "dense_row":
        return np.concatenate([[n], np.minimum(_poisson_quantiles(POISSON_MEAN, m - 1), n)])
    if kind == "empty_rows":
        full = max(1, m // 10)
        return np.concatenate([np.minimum(_poisson_quantiles(POISSON_MEAN, full), n),
                               np.zeros(m - full, np.int64)])
    raise ValueError(kind)


def _nnz(c):
    kind = c["kind"]
    if kind == "stencil2d":
        nx, ny = c["nx"], c["ny"]
        return nx * ny + 2 * (nx - 1) * ny + 2 * nx * (ny - 1)
    if kind == "stencil3d":
        return (3 * c["nx"] - 2) * (3 * c["ny"] - 2) * (3 * c["nz"] - 2)
    m, n = _rows_cols(c)
    if kind == "blockdiag":
        last = m % BLOCK
        return (m // BLOCK) * BLOCK * BLOCK + last * last
    return int(_lengths(kind, m, n).sum())


def _members(c):
    """The batch's matrices: row counts log-uniform in [1,000, 200,000], kinds in turn."""
    out = []
    for i in range(c["count"]):
        # a permutation of the quantiles, so that neighbours differ in size and kind
        q = ((i * 37) % c["count"] + 0.5) / c["count"] if c["count"] % 37 else (i + 0.5) / c["count"]
        m = int(round(math.exp(math.log(1_000) + q * math.log(200))))
        kind = BATCH_KINDS[i % len(BATCH_KINDS)]
        d = {"kind": kind}
        if kind == "stencil2d":
            d["nx"] = max(1, int(round(m ** 0.5)))
            d["ny"] = max(1, int(round(m / d["nx"])))
        elif kind == "stencil3d":
            d["nx"] = d["ny"] = max(1, int(round(m ** (1 / 3))))
            d["nz"] = max(1, int(round(m / (d["nx"] * d["ny"]))))
        else:
            d["m"] = d["n"] = m
        out.append(d)
    return out


def work(case):
    """Each of val, col_idx, row_ptr and x read once, y written once; one multiply-add per
    non-zero and right-hand side."""
    if case["use"] == "batch":
        k = case["k"]
        ms = _members(case)
        nnz = sum(_nnz(d) for d in ms)
        m = sum(_rows_cols(d)[0] for d in ms)
        n = sum(_rows_cols(d)[1] for d in ms)
        return {"bytes": nnz * 8 + 4 * (m + 1) + 4 * k * (m + n), "flops": 2 * nnz * k}
    m, n = _rows_cols(case)
    nnz = _nnz(case)
    s_val = {"f64": 8, "f32": 4, "mixed_f32": 4, "mixed_bf16": 2}[case["vt"]]
    s_vec = 8 if case["vt"] == "f64" else 4
    return {"bytes": nnz * (s_val + 4) + 4 * (m + 1) + s_vec * (m + n), "flops": 2 * nnz}


# --- inputs, on the GPU, from the seed -------------------------------------------------------
def _uniform(count, g, lo, hi):
    return torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _grid_matrix(c, g):
    """5-point (2D) or 27-point (3D) stencil: columns ascending within a row."""
    m, _ = _rows_cols(c)
    r = torch.arange(m, device="cuda", dtype=torch.int64)
    nx, ny = c["nx"], c["ny"]
    ix, iy = r % nx, (r // nx) % ny
    if c["kind"] == "stencil2d":
        steps = [(0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0)]
        iz, nz = torch.zeros_like(r), 1
        centre, noise = 4.0, 1e-3
    else:
        steps = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        iz, nz = r // (nx * ny), c["nz"]
        centre, noise = 26.0, 0.01
    ok = torch.empty(m, len(steps), device="cuda", dtype=torch.bool)
    col = torch.empty(m, len(steps), device="cuda", dtype=torch.int32)
    for j, (dz, dy, dx) in enumerate(steps):
        x, y, z = ix + dx, iy + dy, iz + dz
        ok[:, j] = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
        col[:, j] = (r + dz * nx * ny + dy * nx + dx).to(torch.int32)
    lengths = ok.sum(1)
    own = torch.zeros(len(steps), device="cuda", dtype=torch.bool)
    own[steps.index((0, 0, 0))] = True
    diag = own.expand(m, -1)[ok]
    col = col[ok]
    e = _uniform(col.numel(), g, -noise, noise)
    if c["kind"] == "stencil2d":
        val = torch.where(diag, centre, -1.0) + e
    else:
        val = torch.where(diag, centre, -1.0) * (1 + e)
    return lengths, col, val


def _matrix(c, g):
    """(row_ptr int32, col int32, val float64) on the GPU."""
    m, n = _rows_cols(c)
    if c["kind"] in ("stencil2d", "stencil3d"):
        lengths, col, val = _grid_matrix(c, g)
    elif c["kind"] == "blockdiag":
        r = torch.arange(m, device="cuda", dtype=torch.int64)
        lengths = torch.clamp(m - r // BLOCK * BLOCK, max=BLOCK)
        starts = torch.cumsum(lengths, 0) - lengths
        j = torch.arange(int(lengths.sum()), device="cuda", dtype=torch.int64)
        col = (j + torch.repeat_interleave(r // BLOCK * BLOCK - starts, lengths)).to(torch.int32)
        val = _uniform(col.numel(), g, -1, 1)
    else:
        lengths = torch.from_numpy(_lengths(c["kind"], m, n)).cuda()
        lengths = lengths[torch.randperm(m, generator=g, device="cuda")]
        nnz = _nnz(c)
        row = torch.repeat_interleave(torch.arange(m, device="cuda", dtype=torch.int64), lengths)
        key = row * n + torch.randint(n, (nnz,), generator=g, device="cuda")
        key = torch.sort(key).values
        col = (key - row * n).to(torch.int32)
        if c["kind"] == "dense_row":
            whole = lengths[row] == n
            col[whole] = torch.arange(int(whole.sum()), device="cuda", dtype=torch.int32) % n
        del row, key
        val = _uniform(nnz, g, -1, 1)
    row_ptr = torch.zeros(m + 1, device="cuda", dtype=torch.int32)
    row_ptr[1:] = torch.cumsum(lengths, 0).to(torch.int32)
    return row_ptr, col, val


class _HostCSR:
    """A member of a batch, as Batch takes it: host arrays of one matrix."""

    def __init__(self, m, n, row_ptr, col, val):
        self.m, self.n = m, n
        self.row_ptr, self.col, self.val = (t.cpu().numpy() for t in (row_ptr, col, val))

    @property
    def nnz(self):
        return int(self.row_ptr[-1])


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["use"] == "batch":
        parts = [(_rows_cols(d), _matrix(d, g)) for d in _members(case)]
        n = sum(mn[1] for mn, _ in parts)
        return parts, _uniform(n * case["k"], g, -1, 1).float().view(n, case["k"])
    row_ptr, col, val = _matrix(case, g)
    vec = torch.float64 if case["vt"] == "f64" else torch.float32
    x = _uniform(_rows_cols(case)[1], g, -1, 1).to(vec)
    return (row_ptr, col, val.to(STORE[case["vt"]])), x


def prepare(case, seed):
    if case["use"] == "batch":
        parts, x = _inputs(case, seed)
        b = Batch([_HostCSR(m, n, *a) for (m, n), a in parts], k=case["k"])
        return {"batch": b, "x": x, "y": torch.empty(b.m, case["k"], device="cuda")}
    m, n = _rows_cols(case)
    vt = VALUE_TYPES[case["vt"]]
    (row_ptr, col, val), x = _inputs(case, seed)
    if case["use"] == "handle":
        h = sp.BhsparseSpmvCuda(vt)
        y = np.zeros(m, sp.host_dtype(vt))
        x = x.cpu().numpy()
        if h.init_platform() or h.prepare_mem(m, n, col.numel(), row_ptr.cpu().numpy(),
                                              col.cpu().numpy(), val.cpu().numpy(), x, y):
            raise RuntimeError(h.last_error)
        return {"handle": h, "x": x, "y": y}
    y = torch.empty(m, device="cuda", dtype=x.dtype)
    s = tune.choose_schedule(vt, row_ptr, col, val, x, y, n=n)
    p = sp.Plan(vt, m, n, row_ptr, col, None, *s["config"])
    return {"plan": p, "val": val, "x": x, "y": y}


def run(state):
    if "plan" in state:
        state["plan"].execute(state["val"], state["x"], state["y"])
    elif "batch" in state:
        state["batch"].execute(state["x"], state["y"])
    else:
        h = state["handle"]
        if h.set_x(state["x"]) or h.run_benchmark() or h.get_y():
            raise RuntimeError(h.last_error)
    return state["y"]


def _multiply(row_ptr, col, val, x):
    """A.x in 64 bits for x [n, k], by plain torch."""
    lengths = (row_ptr[1:] - row_ptr[:-1]).long()
    row = torch.repeat_interleave(torch.arange(lengths.numel(), device="cuda"), lengths)
    out = []
    for j in range(x.shape[1]):
        y = torch.zeros(lengths.numel(), device="cuda", dtype=torch.float64)
        out.append(y.index_add_(0, row, val.double() * x[:, j].double()[col.long()]))
    return torch.stack(out, 1)


def exact(case, seed):
    if case["use"] == "batch":
        parts, x = _inputs(case, seed)
        ys, at = [], 0
        for (_, n), (row_ptr, col, val) in parts:
            ys.append(_multiply(row_ptr, col, val.float(), x[at:at + n]))
            at += n
        return torch.cat(ys)
    a, x = _inputs(case, seed)
    y = _multiply(*a, x[:, None])[:, 0]
    return y.cpu().numpy() if case["use"] == "handle" else y
