"""GPU parity of the spectral core (spectral.cuh) at the edges of its grids.

The core picks a grid of 32 RG points (RG = 1 .. 8) from the larger band, keeps
a few kernels in flight per CTA and splits the kernels of an image into slices;
the cases sit at the smallest and largest band of each grid, with kernel counts
that leave remainders, and slices summed in the core or by the second kernel.
Oracle: FT_r2c + calcSOCS + FI in FP64 (oracle/klitho_oracle.c).  Tolerance:
1e-5 of the clear-field intensity, the mixed-precision bar.
"""
import numpy as np
import pytest

import klitho as K
import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,nk", [
    (0, 0, 1), (1, 7, 9), (7, 7, 70), (8, 3, 1), (8, 8, 5), (15, 15, 70), (16, 2, 3), (23, 23, 7), (24, 24, 2),
    (31, 31, 5), (5, 32, 3), (39, 39, 4), (40, 40, 3), (47, 47, 2), (48, 1, 3), (55, 55, 2), (56, 56, 1), (63, 63, 3)])
def test_grid_edges(cuda, Nx, Ny, nk):
    import torch
    Lx, Ly = 8 * Nx + 11, 8 * Ny + 10  # the smallest periods, one odd: 4N+1 within half of them
    krn, sc = synth.random_kernels(nk, Nx, Ny, seed=100 * Nx + Ny + nk)
    sc[-1] = -0.25 * sc[-1]  # eigenvalues of any sign
    masks = np.stack([synth.rect_mask(Lx, 3, seed=s, wmin=2, wmax=max(3, min(Lx, Ly) // 3), Ly=Ly) for s in (1, 2)])
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, nk, nsets=1, max_clips=2)
    plan.set_kernels(0, krn, sc)
    md = torch.from_numpy(masks).cuda()
    out = torch.empty((2, 1, Ly, Lx), dtype=torch.float32, device="cuda")
    plan.forward(md, out)
    torch.cuda.synchronize()
    first = out.cpu().numpy()
    plan.forward(md, out)  # the slice counters were left ready
    torch.cuda.synchronize()
    assert np.array_equal(first, out.cpu().numpy())
    plan.close()
    c = (2 * Ny + 1) * (2 * Nx + 1) // 2
    cf = float(np.sum(np.abs(sc.astype(np.float64)) * np.abs(krn[:, c].astype(np.complex128)) ** 2))
    cf = max(cf, float(np.sum(np.abs(sc)) / krn.shape[1]))
    for m in range(2):
        want = O.socs_image(masks[m], krn.astype(np.complex128), sc, Nx, Ny)
        assert np.abs(first[m, 0] - want).max() <= 1e-5 * cf
