"""The work that programs using this library have it do, as cases that can be prepared, run and timed.

Every case goes through the package's public entry points.  The systems come from the library's own
generators (P1 finite elements with a log-normal conductivity), whose right-hand side is b = A x_true in
FP64, so x_true is the exact answer of a solve; x_true is drawn from the seed.

Kinds of case, and what each stands for:
  golden   one small FP64 solve through host arrays with the default (absolute) tolerance: the reference's
           own workload, whose solvers are limited to n <= 1024; latency is all that counts
  field2d  a permuted and reordered 2D system solved to a true residual on device vectors: what a
           simulation does once per step with the matrix kept resident
  volume3d the same on 3D tetrahedra, with the mixed-precision options those systems are run with
  batch    many independent 2D systems of mixed sizes in one call
  learned  a 2D system solved with the learned G^T G preconditioner (inference is part of set-up)
  run_pcg  the one-call entry: CSR on the host in, solution on the host out, set-up included
  spmv     one product with a resident matrix through host vectors
  train    loss and gradient of the preconditioner network on one training system
  order    reverse Cuthill-McKee ordering of an unordered matrix and the symmetric permutation by it
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

import project_xplus_b200 as xp
from project_xplus_b200 import generators as gen
from project_xplus_b200.batch import BatchSolver
from project_xplus_b200.learned import GnnTrainer, load_weights

ROOT = Path(__file__).resolve().parent.parent


def listed():
    return [
        # the reference's default problem size, precision and tolerance
        {"name": "golden_32", "kind": "golden", "side": 32, "sigma": 1.0, "mesh": 0},
        # a time step of a mid-size simulation: too small to fill the chip by itself
        {"name": "field2d_301", "kind": "field2d", "side": 301, "sigma": 1.5, "values": "f32", "mesh": 0},
        # the headline system of the benchmark
        {"name": "field2d_1108", "kind": "field2d", "side": 1108, "sigma": 2.0, "values": "f32", "mesh": 0},
        # the benchmark's 3D system: the largest that is run in earnest, far above what the caches hold
        {"name": "volume3d_128", "kind": "volume3d", "side": 128, "sigma": 1.5, "values": "f32", "mesh": 0},
        # a 3D system of odd size in 16-bit storage
        {"name": "volume3d_67_bf16", "kind": "volume3d", "side": 67, "sigma": 1.5, "values": "bf16", "mesh": 0},
        # an ensemble of independent systems, sides spread over [45, 256]
        {"name": "batch_64", "kind": "batch", "count": 64, "values": "f32", "mesh": 1000},
        # the learned preconditioner on a system outside its training range
        {"name": "learned_600", "kind": "learned", "side": 600, "sigma": 2.0, "mesh": 0},
        # a system that is solved once: upload, set-up, solve, download
        {"name": "run_pcg_400", "kind": "run_pcg", "side": 400, "sigma": 1.0},
        # an operator product on a 3D system
        {"name": "spmv3d_80", "kind": "spmv", "side": 80, "mesh": 0},
        # a training step's gradient at the upper end of the training sizes
        {"name": "train_450", "kind": "train", "side": 450},
        # reordering a system that arrives in random order
        {"name": "order_500", "kind": "order", "side": 500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["golden", "field2d", "field2d", "volume3d", "volume3d", "batch", "learned", "run_pcg", "spmv",
                       "train", "order"])
    mesh = rng.randrange(1000)
    if kind == "golden":
        return {"kind": kind, "side": _log(rng, 10, 32), "sigma": round(rng.uniform(0.5, 1.5), 3), "mesh": mesh}
    if kind == "field2d":
        return {"kind": kind, "side": _log(rng, 64, 1100), "sigma": round(rng.uniform(0.5, 2.0), 3),
                "values": rng.choice(["f32", "f32", "f16", "bf16"]), "mesh": mesh}
    if kind == "volume3d":
        return {"kind": kind, "side": _log(rng, 16, 127), "sigma": round(rng.uniform(0.5, 1.5), 3),
                "values": rng.choice(["f32", "f32", "f16", "bf16"]), "mesh": mesh}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 8, 96), "values": rng.choice(["f32", "f32", "bf16"]), "mesh": mesh}
    if kind == "learned":
        return {"kind": kind, "side": _log(rng, 150, 900), "sigma": round(rng.uniform(0.5, 2.0), 3), "mesh": mesh}
    if kind == "run_pcg":
        return {"kind": kind, "side": _log(rng, 64, 600), "sigma": round(rng.uniform(0.5, 1.5), 3)}
    if kind == "spmv":
        return {"kind": kind, "side": _log(rng, 24, 96), "mesh": mesh}
    if kind == "train":
        return {"kind": kind, "side": _log(rng, 127, 500)}
    return {"kind": kind, "side": _log(rng, 100, 600)}


def _system(case, seed):
    """(dataset, x_true) of a single-system case.  A case with a "mesh" keeps its matrix, as a program keeps the
    handle it made from it, and takes right-hand sides by the seed; the others take new matrices."""
    kind, side = case["kind"], int(case["side"])
    mesh = int(case.get("mesh", seed))
    if kind in ("volume3d", "spmv"):
        return gen.fem3d(side, sigma=float(case.get("sigma", 1.5)), jitter=0.25, seed=mesh, x_seed=seed)
    if kind == "golden":
        return gen.fem2d(side, sigma=float(case["sigma"]), jitter=0.3, seed=mesh, x_seed=seed)
    return gen.fem2d(side, sigma=float(case.get("sigma", 1.5)), jitter=0.3, seed=mesh, perm_seed=mesh + 1,
                     rcm=kind != "order", x_seed=seed)


def _batch_systems(case, seed):
    sides, sigmas = gen.batch_sides(int(case["count"]), 45, 256, seed=3)
    mesh = int(case["mesh"])
    with ThreadPoolExecutor(8) as pool:
        return list(pool.map(lambda k: gen.fem2d(int(sides[k]), sigma=float(sigmas[k]), seed=mesh + k, x_seed=seed + k),
                             range(len(sides))))


@lru_cache(maxsize=1)
def _stream():
    """The program's one stream: device solves follow each other on it."""
    return torch.cuda.Stream()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems = [d for d, _ in _batch_systems(case, seed)]
        s = BatchSolver([(d.row_ptr, d.col_idx, d.values) for d in systems], values_dtype=case["values"])
        s.set_launch(8, 256)
        s.set_resident(True)
        b = torch.from_numpy(np.concatenate([d.b for d in systems])).cuda()
        return {"kind": kind, "solver": s, "b": b, "x": torch.zeros_like(b), "stream": _stream()}
    d, _ = _system(case, seed)
    if kind == "golden":
        return {"kind": kind, "solver": xp.PcgSolver.from_dataset(d, values_dtype="f64", vector_dtype="f64"),
                "b": d.b, "x0": d.x0}
    if kind in ("field2d", "volume3d", "learned"):
        options = {}
        if kind == "volume3d":
            options = {"replace_every": 50, "replace_drop": 1e-4}
        s = xp.PcgSolver.from_dataset(d, values_dtype=case.get("values", "f32"), **options)
        if kind == "learned":
            s.set_gnn()
        b = torch.from_numpy(d.b).cuda()
        return {"kind": kind, "solver": s, "b": b, "x": torch.zeros_like(b), "stream": _stream(),
                "tau": 1e-10 if kind == "volume3d" else 1e-8}
    if kind == "spmv":
        s = xp.PcgSolver.from_dataset(d)
        return {"kind": kind, "solver": s, "x": d.b}
    if kind == "train":
        params, _ = load_weights()
        return {"kind": kind, "seed": seed,
                "trainer": GnnTrainer([(d.row_ptr, d.col_idx, d.values)], params=params, loss="kaporin")}
    return {"kind": kind, "data": d}


def run(state):
    kind = state["kind"]
    if kind == "golden":
        return state["solver"].solve(state["b"], state["x0"]).solution
    if kind in ("field2d", "volume3d", "learned", "batch"):
        x, stream = state["x"], state["stream"]
        with torch.cuda.stream(stream):
            x.zero_()  # the initial guess; the solution replaces it
        state["solver"].solve_device(state["b"], x, tau=state.get("tau", 1e-8), stream=stream)
        return x
    if kind == "run_pcg":
        return xp.run_pcg(state["data"], xp.SolverConfig(tau=1e-8), tau_mode=xp.XPLUS_TAU_REL_TRUE).solution
    if kind == "spmv":
        return state["solver"].spmv(state["x"])
    if kind == "train":
        loss, grad = state["trainer"].loss_grad(0, state["seed"])
        return {"loss": loss, "grad": grad}
    d = state["data"]
    perm, _ = gen.rcm_device(d.row_ptr, d.col_idx)
    row_ptr, col_idx, values = gen.permute_symmetric_device(d.row_ptr, d.col_idx, d.values, perm)
    return {"perm": perm, "row_ptr": row_ptr, "col_idx": col_idx, "values": values}


def work(case):
    """Bytes: the matrix in its stored form, vectors in and out, each once.  Flops: a product with the matrix and
    the vector updates, times the iterations that such a system typically needs (about 5 per grid side to 1e-8 in
    2D, 6 to 1e-10 in 3D, 1.3 with G^T G, which has three products)."""
    kind = case["kind"]
    if kind == "batch":
        ns = [int(s) ** 2 for s in np.exp(np.linspace(math.log(45), math.log(256), int(case["count"])))]
        return {"bytes": sum(n * (6 * 6 + 24) for n in ns), "flops": sum(5 * math.sqrt(n) * n * 24 for n in ns)}
    side = int(case["side"])
    n = side ** 3 if kind in ("volume3d", "spmv") else side ** 2
    off = 14 * n if kind in ("volume3d", "spmv") else 6 * n
    stored = {"f32": 6, "f16": 4, "bf16": 4}[case.get("values", "f32")]
    once = 2 * off + 12 * n
    if kind == "golden":
        return {"bytes": 10 * (off + n) + 24 * n, "flops": 4 * side * once}
    if kind in ("field2d", "volume3d"):
        return {"bytes": stored * off + 24 * n, "flops": (5 if kind == "field2d" else 6) * side * once}
    if kind == "learned":
        return {"bytes": 12 * off + 24 * n, "flops": 1.3 * side * (4 * off + 14 * n)}
    if kind == "run_pcg":
        return {"bytes": 12 * (off + n) + 28 * n, "flops": 5 * side * once}
    if kind == "spmv":
        return {"bytes": 6 * off + 20 * n, "flops": 2 * off + 3 * n}
    if kind == "train":
        # 11 node products and 3 aggregations of width 32, twice again in the backward pass
        return {"bytes": 4 * (2 * off + 3 * n) + 8 * 11618, "flops": 3 * (11 * 2 * 32 * 32 * n + 3 * 64 * off)}
    return {"bytes": 2 * 12 * (off + n) + 16 * n, "flops": 0}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return np.concatenate([x for _, x in _batch_systems(case, seed)])
    d, x_true = _system(case, seed)
    if kind == "order":
        return None  # integers, and values that are only moved
    if kind == "spmv":
        rows = np.repeat(np.arange(d.n), np.diff(d.row_ptr))
        return np.bincount(rows, weights=d.values * d.b[d.col_idx], minlength=d.n)
    if kind == "train":
        return _network(d)
    return x_true


def _network(d, H=32, layers=3):
    """Kaporin loss and gradient of the preconditioner network in FP64, parameters rounded to BF16 as the forward
    pass defines them (node activations are not rounded here)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    with np.load(ROOT / "project_xplus_b200" / "weights" / "gtg_gnn.npz") as z:
        theta = torch.from_numpy(z["params"].astype(np.float32)).bfloat16().double().to(dev).requires_grad_(True)
    shapes = [(H, 2), (H,)] + [(H, H), (H,), (H, H), (H, H)] * layers
    shapes += [(H, H), (H,), (H, H), (H,), (H,), (H,), (1,), (H,), (1,)]
    parts = theta.split([math.prod(s) for s in shapes])
    p = iter([q.view(s) for q, s in zip(parts, shapes)])
    n = d.n
    a = torch.from_numpy(d.values).to(dev)
    col = torch.from_numpy(d.col_idx.astype(np.int64)).to(dev)
    row = torch.repeat_interleave(torch.arange(n, device=dev), torch.from_numpy(np.diff(d.row_ptr).astype(np.int64)).to(dev))
    on = row == col
    diag = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, row[on], a[on])
    rowabs = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, row, a.abs())
    r, c = row[~on], col[~on]
    e = a[~on] / torch.sqrt(diag[r] * diag[c])
    order = torch.argsort(r * n + c)
    r, c, e = r[order], c[order], e[order]
    key = r * n + c
    low = c < r
    i, j, el = r[low], c[low], e[low]
    # pairs of lower edges (i, j), (i, m) of one row whose ends j and m are neighbours
    first = torch.searchsorted(i, torch.arange(n + 1, device=dev))
    pairs = []
    for k in range(1, int((first[1:] - first[:-1]).max().item())):
        s = torch.arange(len(i), device=dev)
        t = s + k
        s = s[t < first[i + 1]]
        t = s + k
        q = j[s] * n + j[t]
        at = torch.searchsorted(key, q).clamp(max=len(key) - 1)
        hit = key[at] == q
        pairs.append((s[hit], t[hit], e[at[hit]]))
    ps, pt, pe = (torch.cat(v) for v in zip(*pairs))
    f = torch.zeros_like(el).index_add_(0, ps, pe * el[pt]).index_add_(0, pt, pe * el[ps])
    ld = diag.log()
    x = torch.stack([ld - ld.mean(), rowabs / diag - 1.0], 1)
    h = torch.relu(x @ next(p).T + next(p))
    for _ in range(layers):
        wa, ba, wl, wu = next(p), next(p), next(p), next(p)
        message = torch.where(low[:, None], (h @ wl.T)[c], (h @ wu.T)[c]) * e[:, None]
        h = h + torch.relu((h @ wa.T + ba).index_add(0, r, message))
    P, bp, Q, c1, c2, w, bw, wd, bwd = p
    edge = torch.relu((h @ P.T + bp)[i] + (h @ Q.T)[j] + el[:, None] * c1 + f[:, None] * c2)
    go = edge @ w + bw
    t = h @ wd + bwd
    gd = t.exp()
    quad = gd * gd
    quad = quad.index_add(0, i, go * go + 2.0 * el * go * gd[i])
    quad = quad.index_add(0, i[ps], 2.0 * pe * go[ps] * go[pt])
    loss = (quad.log() - 2.0 * t).sum() / n
    grad, = torch.autograd.grad(loss, theta)
    return {"loss": loss.item(), "grad": grad.cpu().numpy()}
