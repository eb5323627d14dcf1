"""The host-buffer entry stages its arrays by pieces of 1 MB over host threads:
its result is the device entry's, bit for bit, whatever the arrays' sizes --
within one piece, at its edges, and over several threads (more than 8 MB)."""
import numpy as np
import pytest
import torch

import pbbfmm3d_b200 as fmm

pytestmark = pytest.mark.gpu

PIECE = (1 << 20) // 8  # values of a piece


@pytest.mark.parametrize("Ns,Nf,C", [
    (1, 1, 1),
    (PIECE // 3, PIECE, 1),  # the weights end inside a piece, the result at its edge
    (PIECE // 3 + 1, PIECE + 1, 1),
    (PIECE // 2, 0, 2),  # sources = targets; the weights one whole piece
    (150_001, 70_000, 5),  # several threads for the inputs, one for the result
    (50_000, 200_003, 3),  # one thread
    (50_000, 400_003, 3),  # several for inputs and result
])
def test_same_as_device_entry(Ns, Nf, C):
    rng = np.random.default_rng(7)
    src = rng.random((Ns, 3)) - 0.5
    tgt = rng.random((Nf, 3)) - 0.5 if Nf else src
    w = rng.standard_normal(Ns * C)
    tree = fmm.kernel_ExpCov(1.0, 3, 3, 1e-5, 0, ell=0.3)
    tree.buildFMMTree()
    out = np.zeros(tgt.shape[0] * C)
    fmm.H2_3D_Compute(tree, tgt, src, w, C, out)
    ds = torch.tensor(src, device="cuda")
    dt = torch.tensor(tgt, device="cuda") if Nf else ds
    ref = torch.zeros(C, tgt.shape[0], dtype=torch.float64, device="cuda")
    fmm.compute_device(tree, dt, ds, torch.tensor(w, device="cuda").view(C, Ns), C, ref)
    ref = ref.cpu().numpy().ravel()
    assert np.array_equal(out, ref)
    fmm.H2_3D_Compute(tree, tgt, src, w, C, out)  # adds to what is there
    assert np.array_equal(out, ref + ref)
