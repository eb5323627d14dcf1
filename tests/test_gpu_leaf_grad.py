"""Gradient leaf phase at every leaf size around its lane layouts (1 to 16
targets per pass, larger leaves in passes) and around its 4 columns per pass:
the gradients with respect to both point sets and the transposed product against
dense float64 sums; the kernels' gradients and the interpolation's against the
same sums at the order's accuracy, mixed against float64 within 4e-5 (sums of
terms that cancel; 3e-6 to 1.5e-5 measured)."""
import numpy as np
import pytest

import pbbfmm3d_b200 as fmm
from helpers import make_tree
from test_gpu_leaf_sizes import _per_leaf, cancelling_sources, eight_leaves

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 3, 4, 6])
@pytest.mark.parametrize("size", [1, 2, 4, 7, 16, 17, 40])
def test_leaf_gradients(size, cols):
    import torch

    rng = np.random.default_rng(10 * size + cols)
    tgt = torch.tensor(_per_leaf(rng, [size] * 64), device="cuda")
    src = torch.tensor(_per_leaf(rng, rng.integers(0, 2 * size + 1, 64)), device="cuda")
    w = torch.tensor(rng.standard_normal((cols, src.shape[0])), device="cuda")
    g = torch.tensor(rng.standard_normal((cols, tgt.shape[0])), device="cuda")
    sigma = 0.3
    d = src[None, :, :] - tgt[:, None, :]
    k = torch.exp(-(d * d).sum(-1) / (2 * sigma ** 2))
    m = (g.T @ w) * k / sigma ** 2
    ref = [(m[:, :, None] * d).sum(1), -(m[:, :, None] * d).sum(0), g @ k]
    t = make_tree("GaussSigma", sigma, 1.0, 2, 6, 1e-9, 1)
    t.buildFMMTree()
    got = {}
    for prec in (fmm.PREC_FP64, fmm.PREC_MIXED):
        o = [torch.zeros_like(tgt), torch.zeros_like(src), torch.zeros_like(w)]
        fmm.compute_adjoint_device(t, tgt, src, w, g, cols, grad_target=o[0], grad_source=o[1],
                                   grad_weight=o[2], precision=prec)
        got[prec] = o
    for a, b, r in zip(got[fmm.PREC_FP64], got[fmm.PREC_MIXED], ref):
        n = r.norm()
        # order 6 on cells of a quarter of the box: the interpolation error of
        # the kernel (1e-4) and, differentiated, ten times that
        assert (a - r).norm() < 2e-3 * n
        assert (a - b).norm() < 4e-5 * n
    t.close()


@pytest.mark.parametrize("cols", [1, 4])
@pytest.mark.parametrize("size", [8, 11, 16])
def test_gradient_sums_are_compensated_pair_by_pair(size, cols):
    import torch

    rng = np.random.default_rng(size)
    src, w, bound = cancelling_sources()
    tgt = eight_leaves(rng, size)
    t = make_tree("Laplacian", 0.0, 1.0, 2, 3, 1e-6, 1)
    t.buildFMMTree()
    dev = lambda a: torch.tensor(a, device="cuda")
    d = tgt - src[0]
    r = np.linalg.norm(d, axis=1)
    for prec, tol in ((fmm.PREC_FP64, 1e-11), (fmm.PREC_MIXED, bound + 1e-6)):
        # forward: the targets' gradients sum over the sources
        gt = torch.zeros(len(tgt), 3, dtype=torch.float64, device="cuda")
        fmm.compute_adjoint_device(t, dev(tgt), dev(src), dev(np.tile(w, (cols, 1))),
                                   dev(np.ones((cols, len(tgt)))), cols, grad_target=gt,
                                   precision=prec)
        ref = -cols * w.sum() * d / r[:, None] ** 3
        err = np.linalg.norm(gt.cpu().numpy() - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert err.max() < tol, prec
        # transposed: the same points as targets (the corners keep the box), the
        # weights' gradients sum over them
        many = np.vstack([src, [[-0.22] * 3, [0.22] * 3]])
        g = np.tile(np.append(w, [0.0, 0.0]), (cols, 1))
        gw = torch.zeros(cols, len(tgt), dtype=torch.float64, device="cuda")
        gs = torch.zeros(len(tgt), 3, dtype=torch.float64, device="cuda")
        fmm.compute_adjoint_device(t, dev(many), dev(tgt), dev(np.ones((cols, len(tgt)))), dev(g),
                                   cols, grad_weight=gw, grad_source=gs, precision=prec)
        assert np.abs(gw.cpu().numpy() / (w.sum() / r) - 1).max() < tol, prec
        err = np.linalg.norm(gs.cpu().numpy() - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert err.max() < tol, prec
    t.close()
