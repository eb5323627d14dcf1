"""Binning and cell lists at their edges: one point, every point in one leaf,
more cells than one block of the list kernels covers, and one buffer given as
sources and targets (binned once) against a copy of it (binned twice)."""
import numpy as np
import pytest

import oracle
import pbbfmm3d_b200 as fmm
from helpers import host_ops, make_tree, oracle_ops, rel
from test_gpu_parity import _meta, gpu_tree, phase_by_phase, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [("one", 1, 3), ("one_leaf", 300, 4), ("corners", 8, 5),
                                  ("many_cells", 3000, 5)], ids=lambda c: c[0])
def test_lists_match_oracle(case):
    how, n, level = case
    rng = np.random.default_rng(n)
    p = rng.uniform(-0.5, 0.5, (n, 3))
    if how == "one_leaf":
        p = 1e-3 * p
    if how == "corners":
        p = np.array([[(i >> 2) & 1, (i >> 1) & 1, i & 1] for i in range(8)]) - 0.5
    phase_by_phase(_meta("ExpCov", 0.3, 1.0, level, 3, 1e-4, 1, 2), p, rng.standard_normal(2 * n))


@pytest.mark.parametrize("precision", [fmm.PREC_FP64, fmm.PREC_MIXED])
@pytest.mark.parametrize("cols", [1, 5])
def test_shared_buffer_is_binned_once_with_the_same_result(precision, cols):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    p = torch.rand(5000, 3, generator=gen, device="cuda", dtype=torch.float64)
    w = torch.randn(cols, 5000, generator=gen, device="cuda", dtype=torch.float64)
    t = make_tree("Laplacian", 0.0, 1.0, 4, 3, 1e-4, 1)
    t.buildFMMTree()
    out = [torch.zeros(cols, 5000, device="cuda", dtype=torch.float64) for _ in range(3)]
    launches = fmm.launch_count()
    fmm.compute_device(t, p, p, w, cols, out[0], precision=precision)
    once = fmm.launch_count() - launches
    # a shorter target set in the same buffer is not the shared case
    fmm.compute_device(t, p[:4000], p, w, cols,
                       torch.zeros(cols, 4000, device="cuda", dtype=torch.float64),
                       precision=precision)
    launches = fmm.launch_count()
    fmm.compute_device(t, p, p.clone(), w, cols, out[1], precision=precision)
    assert fmm.launch_count() - launches > once
    fmm.compute_device(t, p, p, w, cols, out[2], precision=precision)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    t.close()


def test_deep_level_lists_match_oracle():
    """Level 8: more counts than one step of the lists' scan covers."""
    rng = np.random.default_rng(8)
    p = rng.uniform(-0.5, 0.5, (3000, 3))
    p[:1500] = 0.2 + 0.01 * rng.standard_normal((1500, 3))
    w = rng.standard_normal(3000)
    meta = _meta("Laplacian", 0.0, 1.0, 8, 2, 1e-2, 1, 1)
    ops = host_ops("Laplacian", 0.0, 1.0, 8, 2, 1e-2, 1)
    t = gpu_tree(meta, ops)
    assert rel(run_gpu(t, p, p, w, 1), oracle.matvec(oracle_ops(ops, meta), p, p, w, 1)) < 1e-12
    t.close()
