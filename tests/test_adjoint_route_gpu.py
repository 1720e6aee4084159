"""GPU parity of the adjoint on both sides of the size from which its image and gradient
run on the tensor cores (64 tiles of 128 image rows), every engine: images 1e-5 of their
maximum, gradients 1e-4 of max |grad|, against the FP64 oracle."""
import numpy as np
import pytest

import klitho as K
import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["auto", "cuda", "tensor"])
@pytest.mark.parametrize("clips,nsets", [(16, 1), (17, 1), (8, 2), (9, 2)])
def test_adjoint_both_sides(cuda, clips, nsets, mode):
    import torch
    L, N, k = 512, 6, 3
    krn, sc = synth.random_kernels(k, N, N, seed=5)
    dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
    sc = (0.6 / dc * sc).astype(np.float32)
    masks = [synth.smooth_mask(L, seed=s, sigma_px=3.0) for s in (3, 4)]
    target = synth.rect_mask(L, 6, seed=4, wmin=4, wmax=100)
    plan = K.SocsPlan(L, L, N, N, k, nsets=nsets, max_clips=clips, adjoint=True)
    plan.set_synthesis(mode)
    for s in range(nsets):
        plan.set_kernels(s, krn, sc)
    md = torch.from_numpy(np.stack([masks[0]] * (clips - 1) + [masks[1]])).cuda()
    td = torch.from_numpy(np.stack([target] * clips)).cuda()
    grad, loss = torch.empty_like(md), torch.empty(clips * nsets, dtype=torch.float64, device="cuda")
    img = torch.empty((clips, nsets, L, L), dtype=torch.float32, device="cuda")
    plan.vjp(md, td, grad, loss, img)
    torch.cuda.synchronize()
    plan.status()
    plan.close()
    for c, m in ((0, masks[0]), (clips - 1, masks[1])):
        lo, gr, I, _ = O.socs_vjp_reference(m, target, krn, sc, N, N)
        gr = nsets * gr  # the gradient of the loss summed over the sets
        for s in range(nsets):
            assert np.abs(img[c, s].cpu().numpy() - I).max() <= 1e-5 * np.abs(I).max()
        assert np.abs(grad[c].cpu().numpy() - gr).max() <= 1e-4 * np.abs(gr).max()
        assert abs(float(loss.reshape(clips, nsets)[c].sum()) - nsets * lo) <= 1e-4 * nsets * lo


@pytest.mark.parametrize("clips,nsets,few", [(16, 1, True), (17, 1, False), (8, 2, True), (9, 2, False)])
def test_auto_takes_the_engine_of_its_size(cuda, clips, nsets, few):
    """Up to 64 tiles the automatic choice gives the CUDA cores' images bit for bit, above
    them others (the tensor cores'; tensor mode has another mask transform too)."""
    import torch
    L, N, k = 512, 6, 3
    krn, sc = synth.random_kernels(k, N, N, seed=5)
    md = torch.from_numpy(np.stack([synth.smooth_mask(L, seed=s, sigma_px=3.0) for s in range(clips)])).cuda()
    td = (md > 0.5).float()
    images = {}
    plan = K.SocsPlan(L, L, N, N, k, nsets=nsets, max_clips=clips, adjoint=True)
    for s in range(nsets):
        plan.set_kernels(s, krn, sc)
    for mode in ("auto", "cuda", "tensor"):
        plan.set_synthesis(mode)
        images[mode] = torch.zeros((clips, nsets, L, L), dtype=torch.float32, device="cuda")
        plan.vjp(md, td, torch.empty_like(md), torch.empty(clips * nsets, dtype=torch.float64, device="cuda"), images[mode])
        torch.cuda.synchronize()
    plan.status()
    plan.close()
    assert not torch.equal(images["cuda"], images["tensor"])
    assert torch.equal(images["auto"], images["cuda"]) == few
