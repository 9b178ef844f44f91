"""Operator apply and material gradient on grids narrower than a block's columns,
which run blocks of one warp or a thread per node, against the SciPy oracle:
widths around a multiple of the columns such a block yields (32; 30 for the
gradient) and at the rules' limits (16, 48; 60), heights that are no multiple of
a tile.  Tolerances as in the
tests of the wide tiles."""
import numpy as np
import pytest
import torch

from conftest import rel, spec_of
from oracle import helmholtz_ref as H
from test_gpu_operator import medium_of, planes, small_record
from test_gpu_tiles import fields

pytestmark = pytest.mark.gpu
GRIDS = [(19, 9, 2, 2), (2051, 8, 3, 3), (31, 16, 2, 2), (33, 17, 2, 3), (21, 30, 1, 0), (18, 31, 2, 4), (517, 32, 30, 4),
         (22, 33, 2, 4), (23, 48, 2, 5), (25, 49, 2, 5), (16, 60, 2, 5), (29, 61, 2, 5), (13, 64, 70, 4)]


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("nz,nx,S,n_pml", GRIDS)
def test_apply_on_narrow_grids(cuda, nz, nx, S, n_pml, adjoint):
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
@pytest.mark.parametrize("nz,nx,S,n_pml", GRIDS)
def test_gradient_on_narrow_grids(cuda, nz, nx, S, n_pml, dtype):
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
