"""The uniform path's transforms and frequency-domain M2L over the instances
their dispatch knows: every column group (1 to 8, and more than 8), every
order (units per CTA and the k3 loops change with it), levels with 2, 4 and 8
parents per side, sparse cells; in float64 against the oracle phase by phase,
in mixed precision within 2e-6 of float64 (the mixed path's bound)."""
import numpy as np
import pytest

import oracle
import pbbfmm3d_b200 as fmm
from helpers import host_ops, make_tree, oracle_ops, rel
from test_gpu_parity import _meta, gpu_tree, phase_by_phase

pytestmark = pytest.mark.gpu


def _points(n, clustered, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-0.5, 0.5, (n, 3))
    if clustered:
        p[: n // 2] = np.clip(0.2 + 0.01 * rng.standard_normal((n // 2, 3)), -0.5, 0.5)
    return p, rng


CASES = ([(3, 3, c, False) for c in (1, 2, 3, 4, 5, 6, 7, 8, 9, 12)] +
         [(n, 3, 1, False) for n in (2, 4, 5, 6, 7, 8, 9)] +
         [(3, 2, 3, False), (4, 4, 2, True), (5, 4, 8, True)])


@pytest.mark.parametrize("case", CASES, ids=["n%d_L%d_C%d%s" % (n, l, c, "_sparse" if s else "")
                                             for n, l, c, s in CASES])
def test_unif_f64_matches_oracle(case):
    order, level, cols, clustered = case
    p, rng = _points(600, clustered, 10 * order + cols)
    phase_by_phase(_meta("ExpCov", 0.3, 1.0, level, order, 1e-5, 0, cols), p,
                   rng.standard_normal(600 * cols))


def _run(t, p, w, cols, precision):
    t.set_precision(precision)
    out = np.zeros(p.shape[0] * cols)
    fmm.H2_3D_Compute(t, p, p, w, cols, out)
    return out


MIXED = ([(3, 4, c, False) for c in (1, 2, 3, 4, 5, 6, 7, 8, 11)] +
         [(n, 3, 1, False) for n in (2, 4, 5, 6, 7, 8, 9)] +
         # tensor cores: 16 and 32 parents per side, orders with 32, 16 and 8 units per CTA
         [(2, 5, 8, False), (5, 5, 8, True), (6, 5, 16, False), (8, 5, 8, True), (4, 6, 8, True)])


@pytest.mark.parametrize("case", MIXED, ids=["n%d_L%d_C%d%s" % (n, l, c, "_sparse" if s else "")
                                             for n, l, c, s in MIXED])
def test_unif_mixed_matches_f64(case):
    order, level, cols, clustered = case
    n = 20000 if level > 4 else 2000
    p, rng = _points(n, clustered, 10 * order + cols)
    w = rng.standard_normal(n * cols)
    t = make_tree("ExpCov", 0.3, 1.0, level, order, 1e-5, 0)
    t.buildFMMTree()
    ref = _run(t, p, w, cols, fmm.PREC_FP64)
    assert rel(_run(t, p, w, cols, fmm.PREC_MIXED), ref) < 2e-6
    t.close()


# The basis of 10 equidistant nodes amplifies rounding: its Lebesgue constant is
# 17.8 (9 nodes: 10.9), cubed 5.7e3 in three dimensions.  Float64: 2^-53 times that,
# for each of the 10 additions of a transform at the sources' and the targets' end
# less what cancels: 16 times (1.3e-12 to 6.9e-12 seen, the same with the
# transforms computed as direct sums).  Mixed: the bound of 2e-6, which
# order 9 keeps, times (17.8 / 10.9)^2 for the basis at both ends.
TOL10_F64 = 16 * 2.0 ** -53 * 17.85 ** 3
TOL10_MIXED = 2e-6 * (17.85 / 10.95) ** 2


@pytest.mark.parametrize("level", [2, 3])
def test_unif_order_10(level):
    p, rng = _points(600, False, level)
    w = rng.standard_normal(600)
    ops = host_ops("ExpCov", 0.3, 1.0, level, 10, 1e-5, 0)
    meta = _meta("ExpCov", 0.3, 1.0, level, 10, 1e-5, 0, 1)
    t = gpu_tree(meta, ops)
    ref = oracle.matvec(oracle_ops(ops, meta), p, p, w, 1)
    assert rel(_run(t, p, w, 1, fmm.PREC_FP64), ref) < TOL10_F64
    assert rel(_run(t, p, w, 1, fmm.PREC_MIXED), ref) < TOL10_MIXED
    t.close()


@pytest.mark.parametrize("order", [9, 10])
def test_unif_tensor_core_levels_of_the_largest_orders(order):
    """Float64 takes these orders a column at a time."""
    n = 3000
    p, rng = _points(n, True, order)
    w = rng.standard_normal((8, n))
    t = make_tree("ExpCov", 0.3, 1.0, 5, order, 1e-5, 0)
    t.buildFMMTree()
    ref = np.concatenate([_run(t, p, w[c], 1, fmm.PREC_FP64) for c in range(8)])
    assert rel(_run(t, p, w.ravel(), 8, fmm.PREC_MIXED), ref) < (2e-6 if order == 9 else TOL10_MIXED)
    t.close()
