"""kl_socs_set_kernels (two planes, as the kernel files hold them) and
kl_socs_set_kernels_c64 (interleaved) put the same kernels into a plan: images and
gradients equal bit for bit, on plans that keep the kernel layout beside the spectral
core's (adjoint above 128 grid points) and on those that do not, for every kernel set.
"""
import ctypes

import numpy as np
import pytest

import klitho as K
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Nx,Ny,nk,nsets", [
    (512, 512, 8, 8, 3, 2), (127, 40, 0, 2, 1, 1), (260, 300, 31, 7, 4, 2), (300, 310, 32, 37, 2, 2), (512, 520, 55, 55, 2, 1), (300, 310, 32, 37, 1, 1)])
def test_planes_and_interleaved(cuda, Lx, Ly, Nx, Ny, nk, nsets):
    import torch
    plans = [K.SocsPlan(Lx, Ly, Nx, Ny, nk, nsets=nsets, max_clips=1, adjoint=True) for _ in range(2)]
    f = ctypes.POINTER(ctypes.c_float)
    for s in range(nsets):
        krn, sc = synth.random_kernels(nk, Nx, Ny, seed=s + Nx)
        dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
        sc = (0.6 / dc * sc).astype(np.float32)
        re, im = np.ascontiguousarray(krn.real, np.float32), np.ascontiguousarray(krn.imag, np.float32)
        K.check(K.lib().kl_socs_set_kernels(plans[0]._h, s, re.ctypes.data_as(f), im.ctypes.data_as(f), sc.ctypes.data_as(f)),
                "kl_socs_set_kernels")
        plans[1].set_kernels(s, krn, sc)
    mask = torch.from_numpy(synth.smooth_mask(Lx, seed=3, sigma_px=3.0, Ly=Ly)).cuda()[None]
    target = torch.from_numpy(synth.rect_mask(Lx, 6, seed=4, wmin=4, wmax=max(5, min(Lx, Ly) // 3), Ly=Ly)).cuda()[None]
    got = []
    for p in plans:
        img = torch.zeros((1, nsets, Ly, Lx), dtype=torch.float32, device="cuda")
        grad, loss = torch.zeros_like(mask), torch.zeros(nsets, dtype=torch.float64, device="cuda")
        p.vjp(mask, target, grad, loss, img)
        torch.cuda.synchronize()
        p.close()
        got.append((img, grad))
    assert float(got[0][0].abs().max()) > 0 and float(got[0][1].abs().max()) > 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
