"""The mixed Chebyshev M2L on the tensor cores over the forms of its levels:
dense ones (combinations of the children), sparse ones (direct lists) and both
in one launch; accumulators of up to 128, 160 and 256 columns; tiles with a
remainder and with one target; transposed operators.  Within 2e-6 of float64,
the mixed path's bound."""
import numpy as np
import pytest

import pbbfmm3d_b200 as fmm
from helpers import make_tree, rel

pytestmark = pytest.mark.gpu


def _points(how, n, rng):
    p = rng.uniform(-0.5, 0.5, (n, 3))
    if how == "half":  # one half of the box empty, but for two points
        p[:, 0] = -np.abs(p[:, 0])
        p[:2, 0] = 0.45
    if how == "clustered":
        p[: n // 2] = np.clip(0.2 + 0.02 * rng.standard_normal((n // 2, 3)), -0.5, 0.5)
    return p


CASES = [
    # kernel, parameter, order, eps, level, columns, points, how
    ("Laplacian", 0.0, 3, 1e-4, 4, 1, 20000, "uniform"),
    ("GaussSigma", 0.25, 4, 1e-6, 3, 64, 3000, "uniform"),
    ("GaussSigma", 0.1, 5, 1e-9, 4, 3, 20000, "half"),
    ("Laplacian", 0.0, 6, 1e-9, 4, 2, 12000, "uniform"),
    ("Laplacian", 0.0, 6, 1e-12, 3, 5, 4000, "uniform"),
    ("Laplacian", 0.0, 4, 1e-5, 5, 1, 30000, "clustered"),
]


@pytest.mark.parametrize("case", CASES, ids=["%s_n%d_L%d_C%d_%s" % (c[0], c[2], c[4], c[5], c[7])
                                             for c in CASES])
def test_mixed_levels_match_f64(case):
    import torch

    kernel, param, order, eps, level, cols, n, how = case
    rng = np.random.default_rng(order * 10 + cols)
    p = torch.tensor(_points(how, n, rng), device="cuda")
    w = torch.tensor(rng.standard_normal((cols, n)), device="cuda")
    t = make_tree(kernel, param, 1.0, level, order, eps, 1)
    t.buildFMMTree()
    assert t.tensor_core_format() == "f16"
    for adjoint in (False, True):
        o = []
        for prec in (fmm.PREC_FP64, fmm.PREC_MIXED):
            out = torch.zeros(cols, n, dtype=torch.float64, device="cuda")
            if adjoint:
                fmm.compute_adjoint_device(t, p, p, None, w, cols, grad_weight=out, precision=prec)
            else:
                fmm.compute_device(t, p, p, w, cols, out, precision=prec)
            o.append(out.cpu().numpy())
        assert rel(o[1], o[0]) < 2e-6
    t.close()
