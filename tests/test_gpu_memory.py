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


def combined_bytes(t, bound=-1):
    """Sets the bound on the arrays of the combinations; the bytes they take."""
    import ctypes

    held = ctypes.c_int64()
    _lib.check(_lib.lib().pbbfmm_debug_combined_bytes(t._h, bound, ctypes.byref(held)))
    return held.value


def coefficient_bytes(t, level, order, cols, width):
    """Moments, locals, proxies and sums of levels 2 to `level`."""
    o = t.get_operators()
    return sum(8 ** l for l in range(2, level + 1)) * cols * width * (
        2 * order ** 3 + o["rf"] + o["rs"])


@pytest.mark.parametrize("precision", [fmm.PREC_FP64, fmm.PREC_MIXED], ids=["f64", "mixed"])
def test_dense_levels_run_without_room_for_combinations(precision):
    """Room for the level arrays but not for the combinations of dense levels:
    the direct lists run.  Room that the combinations of an earlier call hold is
    given back to a call that needs it."""
    level, order, cols, n = 5, 4, 8, 100000
    tol = 1e-13 if precision == fmm.PREC_FP64 else 2e-6
    t = make_tree("Laplacian", 0.0, 1.0, level, order, 1e-5, 1)
    t.buildFMMTree()
    p, w = points(n, 1), weights(cols, n, 2)
    ref = run(t, p, w, precision)
    held = combined_bytes(t)
    needed = coefficient_bytes(t, level, order, cols, 8 if precision == fmm.PREC_FP64 else 4)
    assert held > 1.3 * needed
    t.close()
    import torch

    t = make_tree("Laplacian", 0.0, 1.0, level, order, 1e-5, 1)
    t.buildFMMTree()
    full = fill_but(needed + 200 * MB)
    assert rel(run(t, p, w, precision), ref) < tol
    assert combined_bytes(t) < 200 * MB
    del full
    torch.cuda.empty_cache()
    run(t, p, w, precision)
    assert combined_bytes(t) == held
    # 16 columns: twice the level arrays, in less than what the combinations hold
    w2 = weights(2 * cols, n, 3)
    full = fill_but(needed // 2)
    two = run(t, p, w2, precision)
    assert combined_bytes(t) < held
    del full
    torch.cuda.empty_cache()
    assert rel(run(t, p, w2, precision), two) < tol
    t.close()


# Laplacian, order 4 (r = 48), level 4: bytes of the combinations of one column of
# the deepest level, 512 parents x 27 proxies (mixed: hi and lo parts of 64 values
# and an exponent) and sums
COLUMN = {fmm.PREC_FP64: 512 * 27 * 96 * 8, fmm.PREC_MIXED: 512 * 27 * (2 * 64 * 2 + 4 + 48 * 4)}


@pytest.mark.parametrize("precision", [fmm.PREC_FP64, fmm.PREC_MIXED], ids=["f64", "mixed"])
@pytest.mark.parametrize("cols", [1, 5])
@pytest.mark.parametrize("share", [1.02, 2.02, 0.35, 0.7, 0.13, 0.0],
                         ids=["column", "columns", "third", "two_thirds", "shallow", "none"])
def test_groups_of_combinations(share, cols, precision):
    """Groups of columns, groups of 9 combinations of one column, the direct list
    below that, level by level: equal but for rounding (float32: the direct list's
    against the combinations', each within 1e-6 of float64)."""
    column = COLUMN[precision]
    tol = 1e-13 if precision == fmm.PREC_FP64 else 2e-6
    t = make_tree("Laplacian", 0.0, 1.0, 4, 4, 1e-5, 1)
    t.buildFMMTree()
    p, w = points(20000, 5), weights(cols, 20000, 6)
    ref = run(t, p, w, precision)
    all_held = combined_bytes(t)
    t.close()
    t = make_tree("Laplacian", 0.0, 1.0, 4, 4, 1e-5, 1)
    t.buildFMMTree()
    bound = int(share * column)
    combined_bytes(t, bound)
    assert rel(run(t, p, w, precision), ref) < tol
    held = combined_bytes(t)
    assert held <= bound < all_held or bound >= all_held
    assert (held > 0) == (share > 0)
    g = weights(cols, 20000, 7)
    import torch

    got = []
    for b in (bound, 1 << 40):
        combined_bytes(t, b)
        o = torch.zeros(cols, 20000, dtype=torch.float64, device="cuda")
        fmm.compute_adjoint_device(t, p, p, w, g, cols, grad_weight=o, precision=precision)
        got.append(o.cpu().numpy())
    assert rel(got[0], got[1]) < tol
    t.close()


def test_adjoint_operators_take_the_place_of_combinations():
    """The transposed operators (0.12 GB at order 6) are made at the first adjoint
    call.  Where the combinations of earlier calls hold the memory that they need,
    these give it back; without any, the call is refused and the next one is right."""
    import torch

    cols, n = 8, 20000
    p, w = points(n, 1), weights(cols, n, 2)

    def adjoint(t):
        o = torch.zeros(cols, n, dtype=torch.float64, device="cuda")
        fmm.compute_adjoint_device(t, p, p, w, w, cols, grad_weight=o)
        return o.cpu().numpy()

    def tree():
        t = make_tree("Laplacian", 0.0, 1.0, 4, 6, 1e-7, 1)
        t.buildFMMTree()
        return t

    t = tree()
    ref = adjoint(t)
    t.close()
    t = tree()
    run(t, p, w, fmm.PREC_FP64)
    held = combined_bytes(t)
    assert held > 200 * MB
    spare = torch.empty(cols * n, dtype=torch.float64, device="cuda")  # the gradient's memory
    full = fill_but(40 * MB)
    del spare
    assert rel(adjoint(t), ref) < 1e-13
    assert combined_bytes(t) < held
    del full
    t.close()
    torch.cuda.empty_cache()
    t = tree()
    combined_bytes(t, 0)
    run(t, p, w, fmm.PREC_FP64)
    spare = torch.empty(cols * n, dtype=torch.float64, device="cuda")
    full = fill_but(40 * MB)
    del spare
    with pytest.raises(fmm.FMMError) as e:
        adjoint(t)
    assert e.value.code == _lib.ERR_ALLOC
    del full
    torch.cuda.empty_cache()
    assert rel(adjoint(t), ref) < 1e-13
    t.close()
