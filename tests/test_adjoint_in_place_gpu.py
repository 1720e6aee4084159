"""kl_socs_vjp with an output written over the targets: the targets are finished with
before the gradient (or, one kernel set, the image of the same pixels) is written, on
every route.  Against the same call with buffers of its own; gradients 1e-4 of
max |grad|, images 1e-5 of their maximum, losses 1e-5 (the routes of the two calls may
differ in rounding).
"""
import numpy as np
import pytest

import klitho as K
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", ["grad", "images", "grad_part"])
@pytest.mark.parametrize("Lx,Ly,Nx,Ny,clips", [
    (512, 512, 8, 8, 1), (127, 40, 7, 2, 2), (254, 65, 15, 3, 1), (252, 64, 15, 3, 1), (1000, 744, 15, 11, 2)])
def test_output_over_targets(cuda, Lx, Ly, Nx, Ny, clips, over):
    import torch
    krn, sc = synth.random_kernels(3, Nx, Ny, seed=Lx + Ly)
    dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, 3, max_clips=clips, adjoint=True)
    plan.set_kernels(0, krn, (0.6 / dc * sc).astype(np.float32))
    masks = torch.from_numpy(np.stack([synth.smooth_mask(Lx, seed=s, sigma_px=3.0, Ly=Ly) for s in range(clips)])).cuda()
    target = torch.from_numpy(np.stack([synth.rect_mask(Lx, 6, seed=4 + s, wmin=4, wmax=max(5, min(Lx, Ly) // 3), Ly=Ly)
                                        for s in range(clips)])).cuda()
    n = target.numel()

    def run(t, grad, img):
        loss = torch.zeros(clips, dtype=torch.float64, device="cuda")
        plan.vjp(masks, t, grad, loss, img)
        torch.cuda.synchronize()
        return loss

    want_g, want_i = torch.empty_like(masks), torch.empty((clips, 1, Ly, Lx), dtype=torch.float32, device="cuda")
    want_l = run(target, want_g, want_i)
    if over == "grad":
        t = target.clone()
        grad, img = t, None
    elif over == "images":
        t = target.clone()
        grad, img = torch.empty_like(masks), t.view(clips, 1, Ly, Lx)
    else:  # the gradient starts half way through the targets
        room = torch.empty(2 * n, dtype=torch.float32, device="cuda")
        t = room[:n].view_as(target).copy_(target)
        at = n // 2 // 4 * 4
        grad, img = room[at:at + n].view_as(target), None
    loss = run(t, grad, img)
    plan.close()
    assert float((loss - want_l).abs().max()) <= 1e-5 * float(want_l.max())
    assert float((grad - want_g).abs().max()) <= 1e-4 * float(want_g.abs().max())
    if img is not None:
        assert float((img - want_i).abs().max()) <= 1e-5 * float(want_i.abs().max())
