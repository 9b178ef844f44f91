"""One GMRES cycle through the Gram-Schmidt kernels' large tiles (2,048 nodes), the
5-point batch and the dense path, against the restated reference cycle: ragged
last tiles in both directions and 1 to 12 basis vectors, so that every split of
the warps over the vectors runs.

Tolerances: the 5-point cycle as in its other test (1e-5).  The dense cycle's
iterate is a combination of preconditioned vectors that are good to 2e-5 and
operator results good to 3e-6 (their own tests): 1e-4."""
import numpy as np
import pytest
import torch

from conftest import rel, spec_of
from oracle import helmholtz_ref as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("n_slots", [1, 16])
def test_cycle_on_tall_tiles(cuda, adjoint, n_slots):
    from nsrno_b200 import Geometry, Medium, gmres_batched
    from nsrno_b200.media import blob_record
    from test_gpu_gmres import fft_preconditioner
    rec = blob_record(nz=260, nx=300, n_pml=20, n_rx=40)
    med = Medium(Geometry.from_record(rec), rec.c, rec.rho, rec.alpha, device=cuda)
    a, b, t = med.coef64.cpu().numpy()
    f, k = 1.5e6, 16
    rng = np.random.default_rng(4)
    g = (rng.standard_normal((2, rec.nz, rec.nx)) + 1j * rng.standard_normal((2, rec.nz, rec.nx))).astype(np.complex64)
    A = H.operator_planes(spec_of(rec), a, b, t, f) * rec.h ** 2
    M = fft_preconditioner(rec, f)
    if adjoint:
        A, forward = A.conj().T.tocsr(), M
        M = lambda v: forward(v.conj()).conj()   # noqa: E731  (the multiplier is even, so M is symmetric)
    rhs = torch.as_tensor(g[np.arange(k) % 2], device=cuda)
    res = gmres_batched(med, [f] * k, rhs=rhs, adjoint=adjoint, tolerance=1e-30, restart=12, max_iterations=12,
                        n_slots=n_slots, return_fields=True, fields_dtype=torch.complex128)
    assert (res.iterations == 12).all()
    for s in (0, 1):
        b_s = g[s].ravel().astype(np.complex128) * rec.h ** 2
        want, _, _ = H.gmres(lambda v: A @ v, b_s, restart=12, max_cycles=1, tolerance=1e-30, precondition=M)
        for q in (s, k - 2 + s):
            assert rel(res.fields[q].cpu().numpy().ravel(), want) < 1e-5
            assert abs(float(res.residual[q]) - H.relative_residual(A, want, b_s)) < 1e-5 * float(res.residual[q])


@pytest.mark.parametrize("adjoint", [False, True])
def test_dense_cycle_on_large_tiles(cuda, adjoint):
    """26 fields of 160 x 224: more nodes than 444 tiles of 2,048."""
    from nsrno_b200.dense import DenseSystem, solve
    from oracle import dense_ref as D
    from test_gpu_tiles import dense_case
    spec, g, medium, alpha, rng = dense_case(96, 160, 12)
    n = 26
    assert n * g.H * g.W > 444 * 2048
    s, o = DenseSystem(g, medium, alpha, 4.3e6, device=cuda), D.DenseSystem(D.DenseGeometry(spec), medium, alpha, 4.3e6)
    inner = (slice(None), slice(g.pz, g.pz + g.h), slice(g.px, g.px + g.w))
    rhs = np.zeros((n, g.H, g.W), complex)
    rhs[inner] = rng.standard_normal((n, g.h, g.w)) + 1j * rng.standard_normal((n, g.h, g.w))

    def each(fn):
        return lambda v: np.stack([fn(p) for p in v.reshape(n, g.H, g.W)]).ravel()
    want, _, _ = H.gmres(each(o.adjoint if adjoint else o.apply), rhs.ravel(), restart=10, max_cycles=1, tolerance=1e-30,
                         precondition=each(lambda p: o.fixed_preconditioner(p, adjoint=adjoint)))
    x, info = solve(s, torch.as_tensor(rhs, device=cuda), adjoint=adjoint, tolerance=1e-30, restart=10, max_cycles=1)
    assert info["steps"] == 10
    assert rel(x.cpu().numpy().ravel(), want) < 1e-4
