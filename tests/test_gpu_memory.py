"""Calls on a card whose memory is nearly full: what does not fit is reported or
done without, nothing is lost by it, and the next call is right."""
import numpy as np
import pytest

import pbbfmm3d_b200 as fmm
from helpers import make_tree, rel
from pbbfmm3d_b200 import _lib

pytestmark = pytest.mark.gpu

MB = 1 << 20


def fill_but(leave):
    """A tensor that leaves about `leave` bytes of device memory free."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    n = (torch.cuda.mem_get_info()[0] - leave) // (2 * MB) * (2 * MB)
    return torch.empty(n, dtype=torch.uint8, device="cuda")


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def points(n, seed, sides=1.0):
    import torch

    rng = np.random.default_rng(seed)
    p = sides * rng.uniform(-0.5, 0.5, (n, 3))
    p[0], p[1] = -0.5, 0.5
    return torch.tensor(p, device="cuda")


def run(t, p, w, precision):
    import torch

    out = torch.zeros(w.shape[0], p.shape[0], dtype=torch.float64, device="cuda")
    fmm.compute_device(t, p, p, w, w.shape[0], out, precision=precision)
    return out.cpu().numpy()


def weights(cols, n, seed):
    import torch

    rng = np.random.default_rng(seed)
    return torch.tensor(rng.standard_normal((cols, n)), device="cuda")


def test_combined_operators_that_do_not_fit():
    """The mixed path's combined operators take 46 MB at order 6 (r = 120) and
    40 are free, everything else being there already: no call loses memory, and
    once there is room the next one is right."""
    t = make_tree("Laplacian", 0.0, 1.0, 4, 6, 1e-7, 1)
    t.buildFMMTree()
    p, w = points(20000, 1), weights(1, 20000, 2)
    ref = run(t, p, w, fmm.PREC_FP64)  # dense levels: the arrays of the combinations
    few, wf = points(300, 3, 0.1), weights(8, 300, 4)
    run(t, few, wf, fmm.PREC_MIXED)    # direct lists: the proxies of more columns
    full = fill_but(40 * MB)
    before, first = free_bytes(), None
    for _ in range(3):
        try:
            assert rel(run(t, p, w, fmm.PREC_MIXED), ref) < 2e-6
        except fmm.FMMError as e:
            assert e.code == _lib.ERR_ALLOC
        first = free_bytes() if first is None else first
    assert free_bytes() == first and first > before - 8 * MB
    del full
    import torch

    torch.cuda.empty_cache()
    assert rel(run(t, p, w, fmm.PREC_MIXED), ref) < 2e-6
    t.close()
