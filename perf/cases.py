"""The matvecs that a user of this framework runs, as cases for timing and for
comparing two versions of it.

A case names a kernel, an interpolation (Chebyshev with its order and SVD
tolerance, or uniform / FFT), the tree level, the points (sources = targets,
or separate sets; uniform or clustered), the columns (right-hand sides), the
precision of the pass and the entry point: ``device`` (compute_device on CUDA
tensors), ``host`` (H2_3D_Compute on numpy buffers, the reference's own call)
or ``grad`` (autograd.fmm_matvec, forward and backward).

Points lie in the unit cube, a small margin inside it, so that separate
sources stay inside the box that is recentred on the targets.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pbbfmm3d_b200 as fmm
from pbbfmm3d_b200.autograd import fmm_matvec

BOX = 1.0


def _case(name, kernel, param, cheb, order, level, sources, targets, cols, precision,
          entry="device", points="uniform", eps=1e-5, wrt=""):
    """targets = 0: the targets are the sources.  wrt (entry "grad"): which
    gradients the backward pass returns, of t(argets), s(ources), w(eights)."""
    return {"name": name, "kernel": kernel, "param": param, "cheb": cheb, "order": order,
            "eps": eps, "level": level, "sources": sources, "targets": targets, "cols": cols,
            "precision": precision, "entry": entry, "points": points, "wrt": wrt}


def listed():
    return [
        # the reference's example problem (a first program; latency counts)
        _case("laplace_20k_fp64", "Laplacian", 0.0, 1, 4, 4, 20_000, 0, 1, "fp64"),
        # a small covariance matvec inside an iterative solver, one right-hand side
        _case("expcov_30k_mixed", "ExpCov", 0.3, 0, 4, 4, 30_011, 0, 1, "mixed"),
        # separate sources and targets, odd sizes and an odd number of columns
        _case("gauss_two_sets_fp64", "GaussSigma", 0.25, 1, 5, 4, 77_777, 33_331, 3, "fp64",
              eps=1e-6),
        # the reference's call on host buffers, a kriging-sized covariance with several columns
        _case("expcov_host_mixed", "ExpCov", 0.3, 0, 5, 5, 200_003, 0, 3, "mixed", entry="host"),
        # one column of a covariance matvec at a middle size, default precision
        _case("expcov_250k_fp64", "ExpCov", 0.2, 0, 5, 5, 250_000, 0, 1, "fp64"),
        # the benchmark's headline: 1M uniform points, 8 right-hand sides
        _case("expcov_1m_mixed", "ExpCov", 0.3, 0, 5, 6, 1_000_000, 0, 8, "mixed"),
        # the same in the default precision
        _case("expcov_1m_fp64", "ExpCov", 0.3, 0, 5, 6, 1_000_000, 0, 8, "fp64"),
        # one right-hand side of it (a solver's matvec with a single vector)
        _case("expcov_1m_one_col_mixed", "ExpCov", 0.3, 0, 5, 6, 1_000_000, 0, 1, "mixed"),
        # the benchmark's clustered Laplacian, 4M points, tensor-core M2L
        _case("laplace_4m_mixed", "Laplacian", 0.0, 1, 6, 7, 4_000_000, 0, 1, "mixed",
              points="clustered", eps=1e-7),
        # clustered Laplacian in the default precision
        _case("laplace_500k_fp64", "Laplacian", 0.0, 1, 6, 6, 500_000, 0, 1, "fp64",
              points="clustered", eps=1e-7),
        # fitting points and weights: forward and backward, separate sets (the
        # benchmark's differentiation workload at a quarter of its points)
        _case("gauss_grad_mixed", "GaussSigma", 0.1, 1, 5, 5, 250_000, 250_000, 4, "mixed",
              entry="grad", eps=1e-6, wrt="sw"),
        # forward and backward in the default precision, all three gradients, sizes that differ
        _case("laplace_grad_fp64", "Laplacian", 0.0, 1, 4, 4, 30_000, 20_011, 2, "fp64",
              entry="grad", wrt="tsw"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes over the listed range (over their logarithm), the
    tree level from the points per leaf, and no dearer than the listed ones."""
    while True:
        cheb = rng.choice([0, 1])
        kernel = rng.choice(["Laplacian", "GaussSigma", "ExpCov"] if cheb else ["ExpCov", "GaussSigma"])
        param = {"Laplacian": 0.0, "GaussSigma": rng.choice([0.1, 0.25]),
                 "ExpCov": rng.choice([0.2, 0.3])}[kernel]
        order = rng.choice([3, 4, 5, 6])
        entry = rng.choice(["device", "device", "device", "host", "grad"])
        precision = rng.choice(["fp64", "mixed"])
        sources = _log_uniform(rng, 5_000, 2_000_000)
        two = entry == "grad" or rng.random() < 0.3
        targets = max(2_000, int(sources * rng.uniform(0.3, 1.5))) if two else 0
        cols = rng.choice([1, 1, 1, 2, 3, 4, 5, 8, 8, 12, 16])
        points = rng.choice(["uniform", "uniform", "clustered"])
        per_leaf = math.exp(rng.uniform(math.log(3.0), math.log(40.0)))
        level = int(round(math.log(sources / per_leaf) / math.log(8.0)))
        level = min(7, max(3, level))
        eps = rng.choice([1e-4, 1e-5, 1e-6]) if cheb else 1e-5
        wrt = rng.choice(["sw", "w", "tsw"]) if entry == "grad" else ""
        c = _case("", kernel, param, cheb, order, level, sources, targets, cols, precision,
                  entry, points, eps, wrt)
        del c["name"]
        nt = targets or sources
        cells = 8.0 ** level * 8.0 / 7.0
        # coefficients of all levels (moments, locals, and the far field's two arrays)
        width = 8 if precision == "fp64" else 4
        per_cell = 2 * order ** 3 * 2 if cheb else 2 * order ** 3 + 4 * order * (2 * order - 1) ** 2
        memory = cells * cols * per_cell * width
        passes = 1.0
        if entry == "grad":
            passes += ("s" in wrt or "w" in wrt) + ("t" in wrt)
        rate = 6e12 if precision == "fp64" else 60e12
        pairs = _near_pairs(c)
        far = _occupied(c) * 189.0 * cols * (2.0 * order ** 6 * 0.4 if cheb
                                             else 8.0 * order * (2 * order - 1) ** 2)
        seconds = passes * (far / rate + pairs * (20 + 4 * cols) / (0.2 * rate))
        if entry == "grad":
            seconds += passes * pairs * 40 * cols / (0.1 * rate)
        if memory < 40e9 and seconds < 0.12 and (sources + nt) * cols < 17_000_000:
            return c


def _occupied(c):
    """Cells of all levels that hold points, for points spread evenly over
    the volume that they cover (clusters: a fifth of the leaves)."""
    n = (c["sources"] + (c["targets"] or c["sources"])) / 2.0
    total = 0.0
    for l in range(2, c["level"] + 1):
        cells = 8.0 ** l
        reach = cells if c["points"] == "uniform" else 0.2 * cells
        total += reach * (1.0 - math.exp(-n / reach))
    return total


def _near_pairs(c):
    """Ordered (target, source) pairs of the 27 neighbour leaves."""
    ns, nt = float(c["sources"]), float(c["targets"] or c["sources"])
    leaves = 8.0 ** c["level"]
    pairs = 27.0 * ns * nt / leaves
    if c["points"] == "clustered":
        # 90 % in 64 blobs of sigma 0.02: the density of pairs is the integral
        # of the squared Gaussian density, (4 pi sigma^2)^-3/2 per blob pair
        blob = 0.81 / 64.0 * (4.0 * math.pi * 0.02 ** 2) ** -1.5
        pairs *= 0.19 + blob * min(1.0, (leaves ** (1.0 / 3.0) * 0.02 * 2) ** 3)
    return min(pairs, ns * nt)


_tree = {}


def _get_tree(c):
    """The tree a program builds once for its kernel and keeps for every
    matvec after that (new points and weights are binned by each call)."""
    key = tuple(c[k] for k in ("kernel", "param", "cheb", "order", "eps", "level"))
    if key not in _tree:
        for t in _tree.values():
            t.close()
        _tree.clear()
        if c["kernel"] == "Laplacian":
            t = fmm.kernel_Laplacian(BOX, c["level"], c["order"], c["eps"], c["cheb"])
        elif c["kernel"] == "ExpCov":
            t = fmm.kernel_ExpCov(BOX, c["level"], c["order"], c["eps"], c["cheb"], ell=c["param"])
        else:
            t = fmm.kernel_GaussSigma(BOX, c["level"], c["order"], c["eps"], c["cheb"],
                                      sigma=c["param"])
        t.buildFMMTree()
        _tree[key] = t
    return _tree[key]


def _points(gen, n, how):
    """n points in the unit cube, 0.005 inside its faces: uniform, or 90 % in
    64 Gaussian blobs (sigma 0.02, centres uniform in [0.1, 0.9]^3) and 10 %
    uniform, in no order."""
    kw = {"generator": gen, "device": "cuda", "dtype": torch.float64}
    p = torch.rand(n, 3, **kw)
    if how == "clustered":
        centre = 0.1 + 0.8 * torch.rand(64, 3, **kw)
        which = torch.randint(0, 64, (n,), generator=gen, device="cuda")
        blob = (centre[which] + 0.02 * torch.randn(n, 3, **kw)).clamp(0.0, 1.0)
        p = torch.where(torch.rand(n, 1, **kw) < 0.9, blob, p)
    return (0.005 + 0.99 * p).contiguous()


def _inputs(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    source = _points(gen, c["sources"], c["points"])
    target = _points(gen, c["targets"], c["points"]) if c["targets"] else source
    weight = torch.randn(c["cols"], c["sources"], generator=gen, device="cuda", dtype=torch.float64)
    g = None
    if c["entry"] == "grad":
        g = torch.randn(c["cols"], target.shape[0], generator=gen, device="cuda",
                        dtype=torch.float64)
    return target, source, weight, g


def prepare(case, seed):
    target, source, weight, g = _inputs(case, seed)
    prec = fmm.PREC_FP64 if case["precision"] == "fp64" else fmm.PREC_MIXED
    state = {"case": case, "tree": _get_tree(case), "precision": prec}
    if case["entry"] == "host":
        state["tree"].set_precision(prec)
        t = target.cpu().numpy()
        state.update(target=t, source=source.cpu().numpy() if case["targets"] else t,
                     weight=weight.cpu().numpy().ravel())
        return state
    if case["entry"] == "grad":
        target.requires_grad_("t" in case["wrt"])
        source.requires_grad_("s" in case["wrt"])
        weight.requires_grad_("w" in case["wrt"])
        state["g"] = g
    state.update(target=target, source=source, weight=weight)
    return state


def run(state):
    c, tree = state["case"], state["tree"]
    target, source, weight = state["target"], state["source"], state["weight"]
    if c["entry"] == "host":
        out = np.zeros(c["cols"] * target.shape[0])
        fmm.H2_3D_Compute(tree, target, source, weight, c["cols"], out)
        return out
    if c["entry"] == "grad":
        out = fmm_matvec(tree, target, source, weight, precision=state["precision"])
        wrt = [x for x in (target, source, weight) if x.requires_grad]
        return [out.detach(), *torch.autograd.grad(out, wrt, state["g"])]
    out = torch.zeros(c["cols"], target.shape[0], dtype=torch.float64, device="cuda")
    fmm.compute_device(tree, target, source, weight, c["cols"], out, precision=state["precision"])
    return out


def work(case):
    """Bytes: points and weights read, results written.  Flops: one kernel
    evaluation (10) and a multiply-add per column for each near-field pair,
    interpolation at the leaves, and for each cell and column the products
    with its 189 interaction cells -- by the frequency-domain form, 8 flops
    per kept frequency, which is the cheaper of the two."""
    ns, nt, cols, n = case["sources"], case["targets"] or case["sources"], case["cols"], case["order"]
    nk = n * (2 * n - 1) ** 2
    same = not case["targets"]
    bytes_ = 8.0 * (3 * ns + (0 if same else 3 * nt) + ns * cols + nt * cols)
    near = _near_pairs(case)
    far = _occupied(case) * 189.0 * cols * 8.0 * nk
    ends = 2.0 * n ** 3 * cols * (ns + nt)
    flops = near * (10.0 + 2.0 * cols) + far + ends
    if case["entry"] == "grad":
        # the transposed pass, and the gradient of every pair for the points
        wrt = case["wrt"]
        bytes_ += 8.0 * (nt * cols + ns * cols * ("w" in wrt) + 3 * ns * ("s" in wrt)
                         + 3 * nt * ("t" in wrt))
        if "s" in wrt or "w" in wrt:
            flops += far + ends + near * (10.0 + 2.0 * cols)
        flops += near * (20.0 + 6.0 * cols) * (("s" in wrt) + ("t" in wrt))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """float64: sums of hundreds to thousands of terms in another order.
    Mixed: float32 terms with compensated totals; the mixed pass lies 2e-7 to
    8e-7 from the float64 pass over these ranges, and its gradients with
    respect to the points (sums of terms that cancel) 3e-6 to 1.5e-5; four
    times the largest of each."""
    grad = case["entry"] == "grad"
    if case["precision"] == "fp64":
        return {"rel": 1e-12 if grad else 2e-13}
    return {"rel": 6e-5 if grad else 3.2e-6}


def _direct(case, target, source, weight, g):
    """The dense sums in float64, in blocks of targets: f = K w and, with g,
    K^T g and the gradients of sum(g f) with respect to both point sets."""
    name, p = case["kernel"], case["param"]
    nt, ns = target.shape[0], source.shape[0]
    f = torch.empty(weight.shape[0], nt, dtype=torch.float64, device="cuda")
    want = g is not None
    gw, gs, gt = torch.zeros_like(weight), torch.zeros_like(source), torch.zeros_like(target)
    block = max(1, min(nt, 60_000_000 // ns))
    for a in range(0, nt, block):
        t = target[a:a + block]
        d = [t[:, i:i + 1] - source[None, :, i] for i in range(3)]
        r2 = d[0] * d[0]
        r2 += d[1] * d[1]
        r2 += d[2] * d[2]
        if not want:
            d = None
        if name == "Laplacian":  # 1/r, 0 where the points coincide
            k = r2.rsqrt().masked_fill_(r2 == 0, 0.0)
            dk = -k * k * k if want else None  # (dK/dr) / r
        elif name == "ExpCov":
            r = r2.sqrt()
            k = torch.exp(-r / p)
            dk = (-k / (p * r)).masked_fill_(r2 == 0, 0.0) if want else None
        else:
            k = torch.exp(-r2 / (2.0 * p * p))
            dk = -k / (p * p) if want else None
        f[:, a:a + block] = weight @ k.T
        if want:
            gb = g[:, a:a + block]
            gw += gb @ k
            dk *= gb.T @ weight
            for i in range(3):
                m = dk * d[i]
                gt[a:a + block, i] = m.sum(dim=1)
                gs[:, i] -= m.sum(dim=0)
    return f, gt, gs, gw


def exact(case, seed):
    nt = case["targets"] or case["sources"]
    if float(case["sources"]) * nt > (1e11 if case["entry"] == "grad" else 2.6e11):
        return None  # more pairs than the dense sum does in about 20 seconds
    target, source, weight, g = _inputs(case, seed)
    f, gt, gs, gw = _direct(case, target, source, weight, g)
    if case["entry"] == "host":
        return f.cpu().numpy().ravel()
    if case["entry"] == "grad":
        return [f] + [x for x, k in ((gt, "t"), (gs, "s"), (gw, "w")) if k in case["wrt"]]
    return f
