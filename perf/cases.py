"""What a user of this framework has it do, as a list of timed cases.

Every case is a binary sparse matrix (or a batch of them) and the public
entry point that transforms it:

  plan     Plan.execute: the resident plan a program keeps for a matrix
  method   the drop-in methods, one call from the COO matrix to the spectrum
  to_host  Plan.execute_to_host: the spectrum streamed into pinned host memory
  batch    Batch.graph_launch: many uneven matrices replayed as one graph

Matrices follow the shapes of the benchmark workloads: uniform positions,
banded power-law and uniform power-law adjacency, and the batch generator's
log-uniform dimensions and densities.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cuspfft_gb300 as gb
from cuspfft_gb300 import synthetic
from cuspfft_gb300.sparse_fft import Batch, sparse_fft_csc_bluestein_cufft_smooth, sparse_fft_csc_bluestein_mixed_radix


def _single(name, entry, pattern, rows, cols, nnz, policy, exact_phases=False):
    return {"name": name, "entry": entry, "pattern": pattern, "rows": rows, "cols": cols, "nnz": nnz,
            "policy": policy, "exact_phases": exact_phases}


def _batch(name, count, lo, hi, dens_lo, dens_hi, dims_seed, policy):
    return {"name": name, "entry": "batch", "count": count, "lo": lo, "hi": hi, "dens_lo": dens_lo,
            "dens_hi": dens_hi, "dims_seed": dims_seed, "policy": policy}


def listed():
    return [
        # one small matrix at a time (a mesh of a few hundred points): launches and latency
        _single("tiny_301x257", "plan", "uniform", 301, 257, 4000, 7),
        # the small plain workload, 0.5 % dense, smooth column count
        _single("uniform_3001x2048", "plan", "uniform", 3001, 2048, 30_730, 3),
        # the power-of-two method family on ordinary odd sizes
        _single("uniform_6007x5003_pow2", "plan", "uniform", 6007, 5003, 60_000, 2),
        # the exact-phase option with the mixed-radix lengths
        _single("uniform_5501x4603_exact", "plan", "uniform", 5501, 4603, 120_000, 3, True),
        # a Hamiltonian-shaped matrix (prime size, banded, power-law degrees)
        _single("banded_8219", "plan", "banded", 8219, 8219, 242_000, 7),
        # a co-authorship graph, the benchmark's default workload
        _single("powerlaw_16706", "plan", "powerlaw", 16706, 16706, 396_000, 7),
        # the largest graph: 6.5 GB of spectrum, several channels a row
        _single("powerlaw_40421", "plan", "powerlaw", 40421, 40421, 351_000, 7),
        # tall and narrow: more than 65536 rows, 4-byte indices, 64-bit phases
        _single("tall_70001x1201", "plan", "uniform", 70001, 1201, 100_000, 7),
        # the drop-in method as a program linked against the reference calls it, default tile
        _single("method_banded_8219", "method", "banded", 8219, 8219, 242_000, 3),
        # the spectrum wanted on the host
        _single("to_host_8219", "to_host", "banded", 8219, 8219, 242_000, 7),
        # the batched workload: 64 uneven matrices
        _batch("batch_64", 64, 500, 12000, 1e-4, 1e-2, 4, 7),
        # many small matrices
        _batch("batch_256_small", 256, 100, 1000, 1e-3, 3e-2, 11, 7),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan"] * 7 + ["square"] * 2 + ["method", "to_host", "batch"])
    policy = rng.choice([2, 3, 7, 7])
    if kind == "batch":
        small = rng.random() < 0.5
        lo, hi = (100, 1000) if small else (500, 6000)
        dens = (1e-3, 3e-2) if small else (1e-4, 1e-2)
        c = _batch("", rng.randrange(16, 65), lo, hi, dens[0], dens[1], rng.randrange(1 << 20), policy)
    elif kind == "square":
        pattern = rng.choice(["banded", "powerlaw"])
        n = _log_uniform(rng, 1500, 30000)
        c = _single("", "plan", pattern, n, n, int(n * rng.uniform(10, 40)), policy)
    else:
        if rng.random() < 0.15:
            rows, cols = _log_uniform(rng, 50000, 75000), _log_uniform(rng, 200, 2500)
        else:
            rows, cols = _log_uniform(rng, 200, 20000), _log_uniform(rng, 200, 20000)
        dens = math.exp(rng.uniform(math.log(1e-4), math.log(1e-2)))
        nnz = min(1_000_000, max(64, int(rows * cols * dens)))
        exact_phases = kind == "plan" and rng.random() < 0.15
        if kind == "method":
            policy = rng.choice([3, 7])
        c = _single("", "plan" if kind == "plan" else kind, "uniform", rows, cols, nnz, policy, exact_phases)
    del c["name"]
    return c


def _matrices(case, seed):
    if case["entry"] == "batch":
        g = np.random.default_rng(case["dims_seed"])
        dims = synthetic.batch_dims(case["count"], case["lo"], case["hi"], seed=case["dims_seed"])
        out = []
        for i, (r, c, _) in enumerate(dims):
            dens = math.exp(g.uniform(math.log(case["dens_lo"]), math.log(case["dens_hi"])))
            out.append(synthetic.uniform_matrix(r, c, max(1, int(round(r * c * dens))), seed * 100003 + i))
        return out
    n, nnz = case["rows"], case["nnz"]
    if case["pattern"] == "banded":
        return [synthetic.banded_powerlaw(n, nnz, band=min(150, n // 8), max_deg=min(400, n // 4), seed=seed)]
    if case["pattern"] == "powerlaw":
        return [synthetic.uniform_powerlaw(n, nnz, max_deg=min(360, n // 4), seed=seed)]
    return [synthetic.uniform_matrix(n, case["cols"], nnz, seed)]


def prepare(case, seed):
    mats = _matrices(case, seed)
    entry, policy = case["entry"], case["policy"]
    if entry == "method":
        return {"entry": entry, "coo": mats[0], "policy": policy}
    if entry == "batch":
        batch = Batch(mats, length_policy=policy)
        # one buffer for all spectra, each matrix a (rows, pitch) view of it
        sizes = [m.rows * info["output_pitch"] for m, info in zip(mats, batch.infos)]
        flat = torch.zeros(sum(sizes), dtype=torch.complex64, device="cuda")
        batch.set_outputs([v.view(m.rows, -1) for v, m in zip(flat.split(sizes), mats)])
        return {"entry": entry, "batch": batch, "out": flat}
    plan = gb.Plan(mats[0], length_policy=policy, exact_phases=int(case["exact_phases"]),
                   stream_tile_rows=gb.GBSP_STREAM_TILE_AUTO if entry == "to_host" else 0)
    if entry == "to_host":
        out = torch.zeros((mats[0].rows, plan.output_pitch), dtype=torch.complex64).pin_memory()
    else:
        out = plan.empty_output()
    return {"entry": entry, "plan": plan, "out": out}


def run(state):
    entry = state["entry"]
    if entry == "method":
        method = sparse_fft_csc_bluestein_mixed_radix if state["policy"] == 3 else sparse_fft_csc_bluestein_cufft_smooth
        return method(state["coo"]).d_output
    if entry == "batch":
        state["batch"].graph_launch()
    elif entry == "to_host":
        state["plan"].execute_to_host(state["out"])
    else:
        state["plan"].execute(state["out"])
    return state["out"]


def _pitch(cols):
    return (cols // 2 + 1 + 3) // 4 * 4


def _shapes(case):
    """(rows, cols, nnz) of every matrix, nnz as asked of the generator."""
    if case["entry"] != "batch":
        return [(case["rows"], case["cols"], case["nnz"])]
    g = np.random.default_rng(case["dims_seed"])
    dims = synthetic.batch_dims(case["count"], case["lo"], case["hi"], seed=case["dims_seed"])
    return [(r, c, max(1, int(round(r * c * math.exp(g.uniform(math.log(case["dens_lo"]),
                                                               math.log(case["dens_hi"]))))))) for r, c, _ in dims]


def work(case):
    """Bytes: every row index and column offset in, every spectrum out.
    Flops: the real 2-D FFT of the same size, 2.5 N log2 N."""
    nbytes = flops = 0
    for rows, cols, nnz in _shapes(case):
        nbytes += nnz * (2 if max(rows, cols) <= 65536 else 4) + 4 * (cols + 1) + 8 * rows * _pitch(cols)
        flops += 2.5 * rows * cols * math.log2(max(2, rows * cols))
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    outs = []
    for coo in _matrices(case, seed):
        a = torch.zeros((coo.rows, coo.cols), dtype=torch.float64, device="cuda")
        a[torch.from_numpy(coo.row_idx).long().cuda(), torch.from_numpy(coo.col_idx).long().cuda()] = 1.0
        half = coo.cols // 2 + 1
        f = torch.zeros((coo.rows, _pitch(coo.cols)), dtype=torch.complex128, device="cuda")
        # by pieces, so that the work areas of prime lengths stay small
        step = max(1, (1 << 27) // coo.cols)
        for i in range(0, coo.rows, step):
            f[i:i + step, :half] = torch.fft.rfft(a[i:i + step], dim=1)
        del a
        step = max(1, (1 << 27) // coo.rows)
        for j in range(0, half, step):
            k = min(j + step, half)
            f[:, j:k] = torch.fft.fft(f[:, j:k].T.contiguous(), dim=1).T
        outs.append(f)
    return torch.cat([f.reshape(-1) for f in outs]) if case["entry"] == "batch" else outs[0]
