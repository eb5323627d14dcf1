"""The float64 Chebyshev far field at the edges of its kernels' tiles, against
the oracle phase by phase with the same operators: ranks from one group of 8
outputs to three blocks of 128, row counts that leave remainders of the 64-row
tiles, many columns, tiles cut along the offsets and not, sparse cells."""
import numpy as np
import pytest

from test_gpu_parity import _meta, phase_by_phase

pytestmark = pytest.mark.gpu

CASES = [
    # kernel, parameter, order, eps, level, columns, points, clustered
    ("Laplacian", 0.0, 2, 1e-1, 2, 1, 200, False),       # ranks below 8
    ("Laplacian", 0.0, 2, 1e-9, 5, 3, 40000, False),     # whole tiles, offsets not cut
    ("Gaussian", 0.0, 3, 1e-4, 3, 63, 700, False),       # a target's columns span two tiles
    ("Laplacian", 0.0, 3, 1e-12, 4, 5, 900, True),       # 27 outputs, mostly empty cells
    ("GaussSigma", 0.25, 4, 1e-6, 3, 2, 3000, False),
    ("GaussSigma", 0.1, 5, 1e-12, 3, 3, 2500, False),    # 125 outputs: 16 groups
    ("Laplacian", 0.0, 6, 1e-14, 3, 2, 2500, True),      # over 128 outputs: two blocks
    ("Laplacian", 0.0, 7, 1e-13, 3, 1, 400, False),      # rank 328, 343 outputs: three blocks
]


@pytest.mark.parametrize("case", CASES, ids=["%s_n%d_L%d_C%d" % (c[0], c[2], c[4], c[5])
                                             for c in CASES])
def test_cheb_f64_tiles(case):
    kernel, param, order, eps, level, cols, n, clustered = case
    rng = np.random.default_rng(order * 100 + cols)
    p = rng.uniform(-0.5, 0.5, (n, 3))
    if clustered:
        p[: n // 2] = np.clip(0.2 + 0.01 * rng.standard_normal((n // 2, 3)), -0.5, 0.5)
    phase_by_phase(_meta(kernel, param, 1.0, level, order, eps, 1, cols), p,
                   rng.standard_normal(n * cols))
