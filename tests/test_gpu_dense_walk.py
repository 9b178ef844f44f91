"""The dense operator's walk down the rows (large batches whose strips are nearly
full) against the FFT-evaluated oracle: ragged last strips and bands in both
precisions, PML in every strip.  Tolerances as in the operator's other tests
(1e-12; complex64 3e-6)."""
import numpy as np
import pytest
import torch

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,pml,fft,n", [(80, 400, 20, (150, 478), 35), (200, 180, 24, (250, 230), 45),
                                           (81, 290, 24, (157, 390), 99)])
def test_dense_walk(cuda, h, w, pml, fft, n):
    from nsrno_b200.dense import DenseSystem
    from oracle import dense_ref as D
    from test_gpu_tiles import dense_case
    spec, g, medium, alpha, rng = dense_case(h, w, pml, fft)
    assert n * g.H * g.W >= 2500000
    s, o = DenseSystem(g, medium, alpha, 5.1e6, device=cuda), D.DenseSystem(D.DenseGeometry(spec), medium, alpha, 5.1e6)
    p = rng.standard_normal((3, g.H, g.W)) + 1j * rng.standard_normal((3, g.H, g.W))
    pt = torch.as_tensor(p, device=cuda)[np.arange(n) % 3]
    for adj in (False, True):
        want = [(o.adjoint if adj else o.apply)(p[k]) for k in range(3)]
        y = (s.adjoint if adj else s.apply)(pt).cpu().numpy()
        y32 = (s.adjoint if adj else s.apply)(pt.to(torch.complex64)).cpu().numpy()
        for k in (0, 1, n - 1):
            assert rel(y[k], want[k % 3]) < 1e-12
            assert rel(y32[k], want[k % 3]) < 3e-6
