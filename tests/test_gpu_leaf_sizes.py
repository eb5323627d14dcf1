"""One-column leaf phase at every leaf size around its lane layouts (targets per
warp 1, 2, 4, 8, 16; 12 and more take the dense kernel), with empty neighbours,
coincident points, separate sources, both interpolations; float64 against the
oracle, mixed precision within 2e-6 of it."""
import numpy as np
import pytest

import oracle
import pbbfmm3d_b200 as fmm
from helpers import host_ops, oracle_ops, rel
from test_gpu_parity import _meta, gpu_tree, run_gpu

pytestmark = pytest.mark.gpu


def _per_leaf(rng, count):
    """count[leaf] points in each of the 64 leaves of [-0.5, 0.5]^3, and the
    corners, which fix the bounding box."""
    p = []
    for i, n in enumerate(count):
        low = np.array([(i >> 4) & 3, (i >> 2) & 3, i & 3]) * 0.25 - 0.5
        p.append(low + 0.25 * rng.uniform(0.02, 0.98, (n, 3)))
    return np.vstack(p + [np.array([[-0.5] * 3, [0.5] * 3])])


@pytest.mark.parametrize("cheb,order", [(1, 3), (0, 4), (1, 7)])
@pytest.mark.parametrize("size", [1, 2, 3, 4, 5, 8, 9, 11, 12, 33])
def test_leaf_sizes(size, cheb, order):
    rng = np.random.default_rng(size)
    kernel = ("Laplacian", 0.0) if cheb else ("ExpCov", 0.3)
    meta = _meta(kernel[0], kernel[1], 1.0, 2, order, 1e-6, cheb, 1)
    ops = host_ops(meta["kernel"], meta["param"], 1.0, 2, order, 1e-6, cheb)
    t = gpu_tree(meta, ops)
    tgt = _per_leaf(rng, [size] * 64)
    src = _per_leaf(rng, rng.integers(0, 2 * size + 1, 64))
    src[: min(5, len(src))] = tgt[: min(5, len(src))]  # coincident pairs contribute K(0), or 0
    w = rng.standard_normal(len(src))
    ref = oracle.matvec(oracle_ops(ops, meta), tgt, src, w, 1)
    assert rel(run_gpu(t, tgt, src, w, 1), ref) < 1e-12
    t.set_precision(fmm.PREC_MIXED)
    assert rel(run_gpu(t, tgt, src, w, 1), ref) < 2e-6
