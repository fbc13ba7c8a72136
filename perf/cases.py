"""The work this library is used for, as cases to be timed: each goes through a public entry
point of jkogb_b200 on inputs made from a seed.

Kinds of a case:
  solve    one whole step loop on device tensors (step_loop_dev), from Y to A, U, Z, SIGMA:
           the everyday call, at the orders where a solve takes at most a second or so
  advance  the resumable loop (Solver: begin, advance, finish) over the first `steps` steps:
           the way the benchmark runs the large orders, whose whole solve takes a minute
  scored   the loop ranked by the trained network (scorer.Scorer.step_loop_dev), bounded
  batch    many small matrices in one launch (Batch.run), bounded; `gram` 1: the Gram ranking
  weights  one build's pair weights (Handle.weights), the kernel-level entry point

Inputs: "gauss" is iid N(0,1) (complex: Re, Im iid N(0,1/2)) with the first n_plus signs +1,
"graded" is G D with D log-uniform in [lo, 1] and the signs in a seeded permutation, the
inputs of jkogb_b200.gen.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import jkogb_b200 as jk
from jkogb_b200 import scorer


def listed():
    return [
        # the smallest calls: a handful of vertices, all latency (launches, host work)
        dict(name="solve_16", kind="solve", n=16, n_plus=12, cplx=0, form="gauss", lo=1.0),
        # an odd order that fills no tile
        dict(name="solve_97", kind="solve", n=97, n_plus=50, cplx=0, form="gauss", lo=1.0),
        # the 256 workload (192 / 64 signs), an ordinary whole solve
        dict(name="solve_256", kind="solve", n=256, n_plus=192, cplx=0, form="gauss", lo=1.0),
        # complex matrices of an ordinary order (zjk)
        dict(name="zsolve_60", kind="solve", n=60, n_plus=30, cplx=1, form="gauss", lo=1.0),
        # graded input between the small and the large orders
        dict(name="advance_512", kind="advance", n=512, n_plus=256, cplx=0, form="graded", lo=1e-6, steps=300),
        # the benchmark's matrix
        dict(name="advance_2048", kind="advance", n=2048, n_plus=1024, cplx=0, form="graded", lo=1e-6, steps=96),
        # the largest order of the workloads, signs +1 first
        dict(name="advance_4096", kind="advance", n=4096, n_plus=2048, cplx=0, form="graded", lo=1e-10, steps=16),
        # the complex workload
        dict(name="zadvance_1024", kind="advance", n=1024, n_plus=512, cplx=1, form="gauss", lo=1.0, steps=48),
        # the learned ranking on the benchmark's matrix
        dict(name="scored_2048", kind="scored", n=2048, n_plus=1024, cplx=0, form="graded", lo=1e-6, steps=128),
        # the batched solver: a share of the 4096-matrix workload, each matrix bounded
        dict(name="batch_384", kind="batch", count=384, nmin=16, nmax=128, gram=0, steps=400),
        # the same with the Gram ranking, fewer matrices than blocks
        dict(name="batch_gram_100", kind="batch", count=100, nmin=16, nmax=128, gram=1, steps=400),
        # one build's weights at a ragged order (partial tiles), unbalanced signs
        dict(name="weights_1811", kind="weights", n=1811, n_plus=700, cplx=0, form="gauss", lo=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "advance", "advance", "scored", "batch", "weights"])
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 1, 384), nmin=16, nmax=2 * rng.randint(12, 64), gram=rng.randint(0, 1),
                    steps=rng.randint(50, 400))
    if kind == "solve":
        cplx = rng.randint(0, 1)
        n = _log_int(rng, 5, 100 if cplx else 256)
    elif kind == "weights":
        cplx, n = 0, _log_int(rng, 100, 2600)
    else:
        cplx = rng.randint(0, 1)
        n = _log_int(rng, 130, 1024 if cplx else 3000)
    graded = rng.randint(0, 1)
    c = dict(kind=kind, n=n, n_plus=max(1, min(n - 1, int(round(n * rng.uniform(0.2, 0.8))))), cplx=cplx,
             form="graded" if graded else "gauss", lo=10.0 ** -rng.randint(2, 10) if graded else 1.0)
    if kind in ("advance", "scored"):
        c["steps"] = max(4, min(300, int(96 * (1.6e9 if cplx else 8.6e9) / float(n) ** 3)))
    return c


def _matrix(case, seed):
    r = np.random.Generator(np.random.PCG64(int(seed)))
    n, n_plus = case["n"], case["n_plus"]
    Y = r.standard_normal((n, n))
    if case["cplx"]:
        Y = math.sqrt(0.5) * (Y + 1j * r.standard_normal((n, n)))
    J = np.concatenate([np.ones(n_plus, np.int64), -np.ones(n - n_plus, np.int64)])
    if case["form"] == "graded":
        Y = Y * np.exp(r.uniform(math.log(case["lo"]), 0.0, n))[None, :]
        # the workloads: random signs, except the largest order's, which has its +1 first
        if n < 4096:
            J = J[r.permutation(n)]
    return Y, J


def _batch(case, seed):
    # the orders belong to the case, the matrices and signs to the seed
    orders = 2 * np.random.Generator(np.random.PCG64(4)).integers(case["nmin"] // 2, case["nmax"] // 2 + 1, case["count"])
    r = np.random.Generator(np.random.PCG64(int(seed)))
    mats, Js = [], []
    for n in orders.tolist():
        mats.append(r.standard_normal((n, n)))
        Js.append(np.where(r.uniform(size=n) < r.uniform(0.2, 0.8), 1, -1).astype(np.int64))
    return mats, Js


def prepare(case, seed):
    s = dict(case=case)
    if case["kind"] == "batch":
        A, J, n, _ = jk.batch_pack(*_batch(case, seed))
        s["A0"] = torch.from_numpy(A).cuda()
        for k in ("A", "U", "Z"):
            s[k] = torch.empty_like(s["A0"])
        s["sigma"] = torch.empty(int(n.sum()), dtype=torch.float64, device="cuda")
        s["info"] = torch.empty(len(n), dtype=torch.int32, device="cuda")
        s["plan"] = jk.Batch(n, np.zeros(len(n), np.int32), J, max_steps=case["steps"])
        if case["gram"]:
            s["scorer"] = scorer.Scorer(None, stall_k=8)
            s["plan"].set_scorer(s["scorer"])
        return s
    Y, J = _matrix(case, seed)
    n = case["n"]
    # column-major, as the entry points take them
    s["Y"] = torch.from_numpy(np.ascontiguousarray(Y.T)).cuda().t()
    s["J"] = J
    if case["kind"] == "weights":
        s["handle"] = jk.Handle(n, J, complex_=bool(case["cplx"]))
        s["W"] = torch.empty((n, n), dtype=torch.float64, device="cuda")
        return s
    for k in ("A", "U", "Z"):
        s[k] = torch.empty((n, n), dtype=s["Y"].dtype, device="cuda").t()
    s["sigma"] = torch.empty(n, dtype=torch.float64, device="cuda")
    if case["kind"] == "advance":
        s["solver"] = jk.Solver(n, J, complex_=bool(case["cplx"]))
    if case["kind"] == "scored":
        s["scorer"] = scorer.Scorer(scorer.load_params(), stall_k=8)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "weights":
        s["handle"].weights(s["Y"].data_ptr(), s["W"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        s["W"].fill_diagonal_(float("nan"))  # a weight matrix has no diagonal
        return s["W"]
    if kind == "batch":
        s["A"].copy_(s["A0"])
        s["plan"].run(*(s[k].data_ptr() for k in ("A", "U", "Z", "sigma", "info")),
                      torch.cuda.current_stream().cuda_stream)
        return {k: s[k] for k in ("info", "A", "U", "Z", "sigma")}
    s["A"].copy_(s["Y"])  # the loop overwrites its matrix
    out = {k: s[k] for k in ("A", "U", "Z", "sigma")}
    if kind == "solve":
        out["info"] = jk.step_loop_dev(s["A"], s["U"], s["Z"], s["sigma"], s["J"])
    elif kind == "scored":
        out["info"], out["exact_steps"] = s["scorer"].step_loop_dev(s["A"], s["U"], s["Z"], s["sigma"], s["J"],
                                                                    max_steps=case["steps"])
    else:
        v = s["solver"]
        v.begin(s["U"].data_ptr(), s["A"].data_ptr(), s["Z"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        v.advance(case["steps"])
        out["info"] = v.finish(s["sigma"].data_ptr())
    return out


def work(case):
    """Per step: A, U and Z read and written once; for every hyperbolic pair the product of its
    two columns (2 operations per row), for every rotated column pair of A, U and Z and every
    rotated row pair of A three operations per entry (8 times that for complex entries).  A
    whole solve takes about 9.4 n steps (the median of random inputs)."""
    def step(n, n_plus, c):
        return 48.0 * n * n * c, (4 if c == 2 else 1) * (2.0 * n * n_plus * (n - n_plus) + 12.0 * n * n)
    if case["kind"] == "batch":
        # even orders spread evenly over [nmin, nmax]: the mean of a step's bytes and operations
        ns = range(case["nmin"], case["nmax"] + 1, 2)
        per = [(step(n, n // 2, 1), min(case["steps"], 9.4 * n)) for n in ns]
        # a matrix goes in, and A, U, Z come out once: a step's bytes need not leave the chip
        return dict(bytes=case["count"] * sum(32.0 * n * n for n in ns) / len(ns),
                    flops=case["count"] * sum(f * m for (_, f), m in per) / len(per))
    n, c = case["n"], 1 + case["cplx"]
    if case["kind"] == "weights":
        return dict(bytes=16.0 * n * n, flops=2.0 * n * case["n_plus"] * (n - case["n_plus"]))
    steps = case.get("steps") or 9.4 * n
    b, f = step(n, case["n_plus"], c)
    return dict(bytes=steps * b, flops=steps * f)


def _exact_weights(Y, J):
    """The weights from their definition: the reduction of the off-diagonal's square norm."""
    A = torch.from_numpy(Y).cuda()
    n = A.shape[0]
    d = torch.diagonal(A)
    app, aqq, apq, aqp = d[:, None], d[None, :], A, A.t()
    w = apq ** 2 + aqp ** 2
    # hyperbolic pairs: the tangent that makes the two columns of the 2x2 block orthogonal,
    # cut to 0.75 (then the block is not diagonalised and keeps off-diagonal entries)
    b = app * apq + aqp * aqq
    n1, n2 = app ** 2 + aqp ** 2, apq ** 2 + aqq ** 2
    m = n1 + n2
    t = -2 * b / (m + torch.sqrt(torch.clamp(m * m - 4 * b * b, min=0.0)))
    cut = t.abs() >= 0.75
    t = torch.where(cut, 0.75 * torch.sign(t), t)
    a11 = torch.sqrt(torch.maximum(n1, n2))
    x, y = b.abs() / a11 ** 2, (app * aqq - apq * aqp).abs() / a11 ** 2
    t2 = -2 * x * y / ((y - x) * (y + x) + 1)
    tu = t2 / (1 + torch.sqrt(1 + t2 * t2))
    cu, cz = torch.rsqrt(1 + tu * tu), 1 / math.sqrt(1 - 0.75 ** 2)
    m11, m12, m21, m22 = a11 * cu, a11 * (x + tu * y) * cu, -tu * a11 * cu, a11 * (y - tu * x) * cu
    left = (((m21 - 0.75 * m22) * cz) ** 2 + ((m12 - 0.75 * m11) * cz) ** 2) * cut
    ch = torch.rsqrt(1 - t * t)
    sh = t * ch
    A0 = A - torch.diag(d)
    g, cn = A0.t() @ A0, (A0 ** 2).sum(0)
    norms = (cn[:, None] - aqp ** 2) + (cn[None, :] - apq ** 2)
    hyp = w - left - 2 * sh * sh * norms - 4 * ch * sh * g
    Jt = torch.from_numpy(J).cuda()
    w = torch.where(Jt[:, None] == Jt[None, :], w, hyp)
    w.fill_diagonal_(float("nan"))
    return w


def exact(case, seed):
    if case["kind"] == "weights":
        return _exact_weights(*_matrix(case, seed))
    if case["kind"] != "solve":
        return None  # where a bounded loop stands has no value of its own
    # Y J Y^H has the eigenvalues J_i sigma_i^2; a converged loop leaves them descending over
    # the +1 signs and ascending over the -1 signs
    Y, J = _matrix(case, seed)
    lam = np.linalg.eigvalsh((Y * J[None, :]) @ Y.conj().T)
    sigma = np.empty(case["n"])
    p = case["n_plus"]
    sigma[J == 1] = np.sqrt(np.abs(np.sort(lam)[::-1][:p]))
    sigma[J == -1] = np.sqrt(np.abs(np.sort(lam)[::-1][p:]))
    return dict(info=None, A=None, U=None, Z=None, sigma=torch.from_numpy(sigma))
