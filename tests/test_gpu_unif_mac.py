"""The uniform path's transforms and frequency-domain M2L over the instances
their dispatch knows: every column group (1 to 8, and more than 8), every
order (units per CTA and the k3 loops change with it), levels with 2, 4 and 8
parents per side, sparse cells; in float64 against the oracle phase by phase,
in mixed precision within 2e-6 of float64 (the mixed path's bound)."""
import numpy as np
import pytest

import pbbfmm3d_b200 as fmm
from helpers import make_tree, rel
from test_gpu_parity import _meta, phase_by_phase

pytestmark = pytest.mark.gpu


def _points(n, clustered, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-0.5, 0.5, (n, 3))
    if clustered:
        p[: n // 2] = np.clip(0.2 + 0.01 * rng.standard_normal((n // 2, 3)), -0.5, 0.5)
    return p, rng


CASES = ([(3, 3, c, False) for c in (1, 2, 3, 4, 5, 6, 7, 8, 9, 12)] +
         [(n, 3, 1, False) for n in (2, 4, 5, 6, 7, 8)] +
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
         [(n, 3, 1, False) for n in (2, 4, 5, 6, 7, 8)] +
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
