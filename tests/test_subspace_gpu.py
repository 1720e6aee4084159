"""GPU parity of the blocked subspace iteration (eigen.cu) over block widths.

The iteration's products and Cholesky factors change kernels with the block
width (multiples of 16 up to 64 columns, wider ones); sources of more than 256
points take it.  Oracle: numpy's eigh of A A^H, A the plan's own FP32 factor
(kl_tcc_factor), so that only the eigensolve is compared.  Eigenvalues to 1e-10
of the largest (FP64 products of the same factor); kernels by the residual
|T v - w v|, 1e-6 of the largest eigenvalue: their float32 storage alone gives
6e-8 sqrt(N) / 2.
"""
import numpy as np
import pytest

import klitho as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nk,block", [
    (512, 1, 3), (512, 4, 15), (512, 8, 16), (512, 9, 17), (512, 20, 33), (512, 24, 0), (512, 24, 49), (512, 30, 64),
    (512, 30, 65), (700, 40, 0), (1100, 24, 0)])
def test_block_widths(cuda, L, nk, block):
    import torch
    src = K.createSource(41, "Annular", 0.6, 0.9)
    rng = np.random.default_rng(L + nk)
    src = (src * rng.uniform(0.5, 1.0, src.shape)).astype(np.float32)  # distinct eigenvalues
    tp = K.TccPlan(src, 1.35, 0.3, L, L, n_medium=1.44)
    assert tp.S > 256
    A = torch.view_as_complex(tp.factor()).cpu().numpy().astype(np.complex128)
    krn, sc, ev, it = tp.topk(nk, block)
    tp.close()
    T = A @ A.conj().T
    w = np.linalg.eigvalsh(T)[::-1][:nk]
    assert it >= 1
    assert np.abs(ev - w).max() <= 1e-10 * w[0]
    v = krn[:, ::-1].T.astype(np.complex128)
    assert np.abs(np.linalg.norm(v, axis=0) - 1).max() <= 1e-5
    assert np.linalg.norm(T @ v - v * w, axis=0).max() <= 1e-6 * w[0]
