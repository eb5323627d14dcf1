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


def cancelling_sources(tiles=4):
    """Sources at one point, in a leaf that neighbours all others, with weights
    whose products with one kernel value are exact: of 32 in a row two large
    ones, 28 ones and the negatives of the large ones.  Returns them with the
    bound on a compensated sum's relative error (twice the unit roundoff times
    sum |x| / |sum x|, to first order); plain float32 sums of such a row lose
    up to 2e-4."""
    w = np.ones(32)
    w[:2], w[30:] = 4096.0, -4096.0
    bound = 2.0 * 2.0 ** -24 * np.abs(w).sum() / abs(w.sum())
    w = np.tile(w, tiles)
    return np.tile([[0.05, 0.07, 0.03]], (w.size, 1)), w, bound


def eight_leaves(rng, per_leaf):
    """per_leaf points in each of the eight leaves around the centre of a
    level-2 tree (no far field between them), the first and last at the corners
    that centre the box."""
    p = []
    for i in range(8):
        low = np.array([(i >> 2) & 1, (i >> 1) & 1, i & 1]) * 0.22 - 0.21
        p.append(low + rng.uniform(0.0, 0.2, (per_leaf, 3)))
    p[0][0], p[7][-1] = -0.22, 0.22
    return np.vstack(p)


@pytest.mark.parametrize("size", [5, 8, 11])
def test_one_column_sums_are_compensated_pair_by_pair(size):
    rng = np.random.default_rng(size)
    src, w, bound = cancelling_sources()
    tgt = eight_leaves(rng, size)
    t = gpu_tree(_meta("Laplacian", 0.0, 1.0, 2, 3, 1e-6, 1, 1))
    ref = w.sum() / np.linalg.norm(tgt - src[0], axis=1)
    assert np.abs(run_gpu(t, tgt, src, w, 1) / ref - 1).max() < 1e-11
    t.set_precision(fmm.PREC_MIXED)
    # beside the sum, the rounding of the kernel value itself (a few ulps)
    assert np.abs(run_gpu(t, tgt, src, w, 1) / ref - 1).max() < bound + 5e-7
    t.close()
