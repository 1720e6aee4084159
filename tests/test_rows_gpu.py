"""GPU parity of the row transforms by matrix products (socs_rows.cu): widths with
0 to 2 factors of two, edges of their tiles (64 pixels and their mirrors, 32 and 64
rows, 16 bins per thread group), many and few rows.  Forward against the FP64 oracle,
1e-5 of clear field; adjoint against torch complex128 autograd, 1e-4 of max |grad|
(the bars of the general pipeline), with and without an image output.
"""
import numpy as np
import pytest

import klitho as K
import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Nx,Ny,clips", [
    (127, 40, 7, 2, 1), (129, 33, 8, 2, 2), (254, 65, 15, 3, 1), (257, 64, 16, 3, 3), (262, 31, 31, 1, 1), (381, 96, 23, 5, 2),
    (450, 70, 55, 4, 1), (131, 1100, 4, 9, 9), (500, 100, 20, 4, 2), (1002, 50, 13, 3, 1)])
def test_forward(cuda, Lx, Ly, Nx, Ny, clips):
    import torch
    krn, sc = synth.random_kernels(3, Nx, Ny, seed=Lx + Ly)
    masks = np.stack([synth.smooth_mask(Lx, seed=s, sigma_px=3.0, Ly=Ly) for s in range(clips)])
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, 3, max_clips=clips)
    assert plan.engine == "general"
    plan.set_kernels(0, krn, sc)
    out = torch.empty((clips, 1, Ly, Lx), dtype=torch.float32, device="cuda")
    plan.forward(torch.from_numpy(masks).cuda(), out)
    got = out.cpu().numpy()
    plan.close()
    cf = float(np.sum(sc.astype(np.float64) * np.abs(krn[:, krn.shape[1] // 2].astype(np.complex128)) ** 2))
    for c in (0, clips - 1):
        want = O.socs_image(masks[c], krn.astype(np.complex128), sc, Nx, Ny)
        assert np.abs(got[c, 0] - want).max() <= 1e-5 * max(cf, np.abs(want).max())


@pytest.mark.parametrize("Lx,Ly,Nx,Ny,clips,with_image", [
    (127, 40, 7, 2, 1, True), (254, 65, 15, 3, 2, False), (263, 64, 32, 4, 1, True), (131, 1100, 4, 9, 9, False),
    (450, 70, 55, 4, 1, True)])
def test_adjoint(cuda, Lx, Ly, Nx, Ny, clips, with_image):
    import torch
    krn, sc = synth.random_kernels(3, Nx, Ny, seed=Lx + Ly)
    dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
    sc = (0.6 / dc * sc).astype(np.float32)
    mask = synth.smooth_mask(Lx, seed=3, sigma_px=3.0, Ly=Ly)
    target = synth.rect_mask(Lx, 6, seed=4, wmin=4, wmax=max(5, min(Lx, Ly) // 3), Ly=Ly)
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, 3, max_clips=clips, adjoint=True)
    plan.set_kernels(0, krn, sc)
    md = torch.from_numpy(np.stack([mask] * clips)).cuda()
    td = torch.from_numpy(np.stack([target] * clips)).cuda()
    grad, loss = torch.empty_like(md), torch.empty(clips, dtype=torch.float64, device="cuda")
    img = torch.empty((clips, 1, Ly, Lx), dtype=torch.float32, device="cuda") if with_image else None
    plan.vjp(md, td, grad, loss, img)
    torch.cuda.synchronize()
    plan.close()
    lo, gr, I, _ = O.socs_vjp_reference(mask, target, krn, sc, Nx, Ny)
    g = grad.cpu().numpy()
    for c in (0, clips - 1):
        assert np.abs(g[c] - gr).max() <= 1e-4 * np.abs(gr).max()
        assert abs(float(loss[c]) - lo) <= 1e-4 * lo
    if with_image:
        assert np.abs(img[0, 0].cpu().numpy() - I).max() <= 1e-5 * np.abs(I).max()
