"""Rounding of the spectral core's sums over kernel slices and residues: the error of one
clip's image against the library's FP64 path, root mean square over three seeds, where
64 kernels of falling weight are split into many slices (added by the core's last CTA and
by the second kernel) and on a grid that is no power of two.

The limits lie between what these shapes showed with the slices added from the largest
kernels on in one chain of 32 bits (2.3e-7, 3.2e-7, 2.8e-7) and with the sums as they are
(1.4e-7, 2.0e-7, 2.3e-7); the warp-FFT kernels before the core showed 2.0e-7, 2.0e-7 and
2.7e-7.
"""
import numpy as np
import pytest

import klitho as K
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,N,limit", [(512, 8, 2.0e-7), (1024, 15, 2.4e-7), (2048, 35, 2.6e-7)])
def test_image_error(cuda, L, N, limit):
    import torch
    nk, e = 64, []
    for seed in (1, 2, 3):
        krn, sc = synth.random_kernels(nk, N, N, seed=seed)
        sc = (np.sort(np.abs(sc))[::-1] * np.exp(-np.arange(nk) / 16.0)).astype(np.float32)
        sc = (0.6 / float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2)) * sc).astype(np.float32)
        mask = torch.from_numpy(synth.rect_mask(L, max(8, L // 40), seed=seed * 10)).cuda()[None]
        plan = K.SocsPlan(L, L, N, N, nk)
        plan.set_kernels(0, krn, sc)
        got = torch.empty((1, 1, L, L), dtype=torch.float32, device="cuda")
        plan.forward(mask, got)
        want = torch.empty((1, L, L), dtype=torch.float64, device="cuda")
        K.fp64_socs_forward(mask, N, N, torch.view_as_real(torch.from_numpy(krn)).cuda().contiguous(),
                            torch.from_numpy(sc).cuda(), want)
        torch.cuda.synchronize()
        plan.close()
        e.append(float((got[:, 0].double() - want).norm() / want.norm()))
    assert np.sqrt(np.mean(np.square(e))) <= limit
