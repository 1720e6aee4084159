"""GPU parity of the row syntheses with factored twiddles (row_fold.cuh): every register
FFT length of theirs (8 to 64 points), lanes with a remainder, bins below, at and above a
multiple of that length, tables in shared memory and beyond its limit.  Against the FP64
oracle: images 1e-5 of their maximum, gradients 1e-4 of max |grad| (the general
pipeline's bars).
"""
import numpy as np
import pytest

import klitho as K
import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Nx,Ny,clips", [
    (264, 40, 2, 2, 1), (264, 33, 4, 2, 3), (1000, 32, 62, 3, 1),         # 8 points; 5, 9, 125 bins
    (528, 64, 7, 3, 2), (560, 35, 40, 2, 1),                              # 16 points
    (1056, 32, 15, 2, 1), (1120, 32, 16, 2, 2), (1056, 300, 47, 3, 5),    # 32 points; 31, 33, 95 bins
    (2112, 32, 31, 2, 1), (2176, 32, 32, 2, 1), (2112, 40, 63, 2, 1),     # 64 points; 63, 65, 127 bins
    (16408, 32, 5, 2, 1), (23168, 32, 21, 2, 1)])                         # tables beyond 96 KB
def test_forward_and_adjoint(cuda, Lx, Ly, Nx, Ny, clips):
    import torch
    krn, sc = synth.random_kernels(3, Nx, Ny, seed=Lx + Ly)
    dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
    sc = (0.6 / dc * sc).astype(np.float32)
    mask = synth.smooth_mask(Lx, seed=3, sigma_px=3.0, Ly=Ly)
    target = synth.rect_mask(Lx, 6, seed=4, wmin=4, wmax=max(5, min(Lx, Ly) // 3), Ly=Ly)
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, 3, max_clips=clips, adjoint=True)
    assert plan.engine == "general"
    plan.set_kernels(0, krn, sc)
    md = torch.from_numpy(np.stack([mask] * clips)).cuda()
    td = torch.from_numpy(np.stack([target] * clips)).cuda()
    grad, loss = torch.empty_like(md), torch.empty(clips, dtype=torch.float64, device="cuda")
    img = torch.empty((clips, 1, Ly, Lx), dtype=torch.float32, device="cuda")
    out = torch.empty_like(img)
    plan.forward(md, out)
    plan.vjp(md, td, grad, loss, img)
    torch.cuda.synchronize()
    plan.close()
    lo, gr, I, _ = O.socs_vjp_reference(mask, target, krn, sc, Nx, Ny)
    for c in (0, clips - 1):
        for got in (out, img):
            assert np.abs(got[c, 0].cpu().numpy() - I).max() <= 1e-5 * np.abs(I).max()
        assert np.abs(grad[c].cpu().numpy() - gr).max() <= 1e-4 * np.abs(gr).max()
        assert abs(float(loss[c]) - lo) <= 1e-4 * lo
