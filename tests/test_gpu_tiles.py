"""The tiled node kernels (operator apply, material gradient) at the edges of
their tiles, against the SciPy oracle: widths around a multiple of 32 and 128,
heights that are no multiple of the tile, both tile heights of the dispatch.

Tolerances: complex128 results differ from the oracle by rounding of some 20
operations, 20 x 1.1e-16 amplified by the cancellation of the flux sum (a
factor of 8 / (k0 h)^2, below 50 here): 1e-13.  The gradient adds up to 20
systems and its own cancellation: 1e-12.  complex64: 20 x 6e-8, 2e-6."""
import numpy as np
import pytest
import torch

from conftest import rel, spec_of
from oracle import helmholtz_ref as H
from test_gpu_operator import medium_of, planes, small_record

pytestmark = pytest.mark.gpu


def fields(S, rec, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((S, rec.nz, rec.nx)) + 1j * rng.standard_normal((S, rec.nz, rec.nx))


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("nz,nx,S,n_pml", [(17, 130, 2, 6), (19, 31, 1, 4), (9, 33, 2, 0), (243, 129, 20, 9)])
def test_apply_tiles(cuda, nz, nx, S, n_pml, adjoint):
    from nsrno_b200 import apply
    rec = small_record(nz=nz, nx=nx, n_pml=n_pml)
    med = medium_of(rec, cuda)
    a, b, t = planes(med)
    freqs = np.linspace(0.9e6, 2.6e6, S)
    x = fields(S, rec, 1)
    y64 = apply(med, torch.as_tensor(x, device=cuda), freqs, adjoint=adjoint).cpu().numpy()
    y32 = apply(med, torch.as_tensor(x.astype(np.complex64), device=cuda), freqs, adjoint=adjoint).cpu().numpy()
    for s in (0, S - 1):
        A = H.operator_planes(spec_of(rec), a, b, t, freqs[s])
        ref = ((A.conj().T.tocsr() if adjoint else A) @ x[s].ravel()) * rec.h ** 2
        assert rel(y64[s].ravel(), ref) < 1e-13
        assert rel(y32[s].ravel(), ref) < 2e-6


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("nz,nx,S,n_pml", [(17, 130, 2, 6), (19, 31, 3, 4), (9, 33, 1, 0), (530, 1030, 2, 24),
                                           (13, 128, 70, 3)])
def test_gradient_tiles(cuda, nz, nx, S, n_pml, dtype):
    from nsrno_b200 import grad_accum
    rec = small_record(nz=nz, nx=nx, n_pml=n_pml)
    med = medium_of(rec, cuda)
    a, b, t = planes(med)
    freqs = np.linspace(0.9e6, 2.6e6, S)
    u, lam = fields(S, rec, 2).astype(dtype), fields(S, rec, 3).astype(dtype)
    gc, gr = grad_accum(med, freqs, torch.as_tensor(u, device=cuda), torch.as_tensor(lam, device=cuda))
    want = [sum(p) for p in zip(*[H.material_gradient_planes(spec_of(rec), a, b, t, f, u[s], lam[s])
                                  for s, f in enumerate(freqs)])]
    assert rel(gc.cpu().numpy(), want[0]) < 1e-12
    assert rel(gr.cpu().numpy(), want[1]) < 1e-12
