"""Calls back to back on a stream of the caller's: each kernel starts ahead of its
predecessor's end (kl_launch.cuh), so a read that comes too early would see the previous
call's data.  Two masks alternate in one buffer, written by a kernel just before each
call, and the kernels are exchanged half way; every output must equal that of the same
call made alone, bit for bit.  Plans of every route: both pipelines, the tensor-core
synthesis, row products, factored rows, odd heights, wide grids.
"""
import numpy as np
import pytest

import klitho as K
import synth

pytestmark = pytest.mark.gpu

ROUTES = [
    # Lx, Ly, Nx, Ny, clips, synthesis
    (512, 512, 8, 8, 1, "auto"), (1024, 1024, 15, 15, 3, "auto"), (512, 512, 8, 8, 2, "tensor"),
    (1000, 744, 15, 11, 2, "auto"), (127, 40, 7, 2, 2, "auto"), (2112, 64, 31, 2, 2, "auto"), (1056, 992, 40, 39, 1, "auto")]
CALLS = 12


def _kernels(nk, Nx, Ny):
    out = []
    for seed in (1, 2):
        krn, sc = synth.random_kernels(nk, Nx, Ny, seed=seed)
        dc = float(np.sum(sc * np.abs(krn[:, krn.shape[1] // 2]) ** 2))
        out.append((krn, (0.6 / dc * sc).astype(np.float32)))
    return out


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("Lx,Ly,Nx,Ny,clips,mode", ROUTES)
def test_back_to_back(cuda, Lx, Ly, Nx, Ny, clips, mode, adjoint):
    import torch
    nk = 5
    kernels = _kernels(nk, Nx, Ny)
    plan = K.SocsPlan(Lx, Ly, Nx, Ny, nk, max_clips=clips, adjoint=adjoint)
    if mode != "auto":
        plan.set_synthesis(mode)
    src = [torch.from_numpy(np.stack([synth.smooth_mask(Lx, seed=10 * m + c, sigma_px=3.0, Ly=Ly) for c in range(clips)])).cuda()
           for m in (0, 1)]
    target = torch.from_numpy(np.stack([synth.rect_mask(Lx, 6, seed=4, wmin=4, wmax=max(5, min(Lx, Ly) // 3), Ly=Ly)] * clips)).cuda()
    masks = torch.empty_like(src[0])
    outs = [[torch.empty((clips, 1, Ly, Lx), dtype=torch.float32, device="cuda"), torch.empty_like(masks)] for _ in range(CALLS)]
    loss = torch.empty(clips, dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()

    def call(m, out):
        torch.mul(src[m], 1.0, out=masks)
        if adjoint:
            plan.vjp(masks, target, out[1], loss, out[0], stream=st)
        else:
            plan.forward(masks, out[0], stream=st)

    want = {}
    for s, (krn, sc) in enumerate(kernels):
        plan.set_kernels(0, krn, sc)
        for m in (0, 1):
            ref = [torch.zeros_like(t) for t in outs[0]]
            torch.cuda.synchronize()
            with torch.cuda.stream(st):
                call(m, ref)
            torch.cuda.synchronize()
            want[s, m] = ref
    assert not torch.equal(want[0, 0][0], want[0, 1][0]) and not torch.equal(want[0, 0][0], want[1, 0][0])
    for s, (krn, sc) in enumerate(kernels):
        plan.set_kernels(0, krn, sc)
        with torch.cuda.stream(st):
            for i in range(CALLS):
                call(i % 2, outs[i])
        st.synchronize()
        for i in range(CALLS):
            assert torch.equal(outs[i][0], want[s, i % 2][0]), (s, i)
            if adjoint:
                assert torch.equal(outs[i][1], want[s, i % 2][1]), (s, i)
    plan.close()
