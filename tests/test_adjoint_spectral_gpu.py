"""GPU parity of the adjoint's spectral core (adjoint_spectral.cu) at the edges of
its grids (32 RG points, RG = 1 .. 4, the larger grids' kernel above), with kernel
counts that leave remainders and two kernel sets.  Reference: torch complex128
autograd of the same loss (oracle.socs_vjp_reference).  Tolerance: 1e-4 of
max |grad|, the adjoint's bar (the resist's slope, alpha = 50, multiplies the FP32
rounding of the image, about 1e-6).  Bands of one or two frequencies are left out:
their images stay away from the threshold, and where the sigmoid s saturates dL/dI
carries the FP32 rounding of 1 - s, 6e-8 / (1 - s) of itself (5e-3 at N = 0).
"""
import numpy as np
import pytest

import klitho as K
import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,nk,nsets", [
    (4, 7, 1, 1), (7, 7, 5, 2), (8, 8, 3, 1), (15, 15, 7, 2), (3, 15, 1, 1), (16, 3, 3, 1), (23, 23, 2, 1), (24, 24, 3, 2),
    (31, 31, 2, 1), (31, 2, 5, 1), (32, 10, 2, 1)])
def test_grid_edges(cuda, Nx, Ny, nk, nsets):
    import torch
    Lx, Ly = 8 * Nx + 11, 8 * Ny + 10
    sets = []
    for s in range(nsets):
        krn, sc = synth.random_kernels(nk, Nx, Ny, seed=31 * Nx + Ny + 7 * s)
        dc = float(np.sum(sc * np.abs(krn[:, (2 * Ny + 1) * (2 * Nx + 1) // 2]) ** 2))
        sets.append((krn, (0.4 / max(dc, 0.05) * sc).astype(np.float32)))
    mask = synth.smooth_mask(Lx, seed=Nx, sigma_px=2.0, Ly=Ly)
    target = synth.rect_mask(Lx, 3, seed=Ny, wmin=2, wmax=max(3, min(Lx, Ly) // 3), Ly=Ly)
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, nk, nsets=nsets, max_clips=2, adjoint=True)
    for s, (krn, sc) in enumerate(sets):
        plan.set_kernels(s, krn, sc)
    md = torch.from_numpy(np.stack([mask, mask])).cuda()
    td = torch.from_numpy(np.stack([target, target])).cuda()
    grad = torch.empty_like(md)
    loss = torch.empty((2, nsets), dtype=torch.float64, device="cuda")
    plan.vjp(md, td, grad, loss, alpha=50.0, threshold=0.225)
    torch.cuda.synchronize()
    plan.close()
    want, wloss = 0.0, []
    for krn, sc in sets:
        lo, gr = O.socs_vjp_reference(mask, target, krn, sc, Nx, Ny)[:2]
        want = want + np.asarray(gr)
        wloss.append(float(lo))
    got = grad.cpu().numpy()
    assert np.array_equal(got[0], got[1])
    assert np.abs(got[0] - want).max() <= 1e-4 * np.abs(want).max()
    assert np.abs(loss.cpu().numpy()[0] - wloss).max() <= 1e-4 * max(wloss)
