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


def dense_case(h, w, pml, fft=None):
    from nsrno_b200.dense import DenseGeometry
    spec = {"medium_shape": [h, w], "dx_m": 5e-5, "x0_m": -0.5 * (w - 1) * 5e-5, "z0_m": -0.0002, "native_dt_s": 2.5e-9,
            "pml": pml, "eta_per_unit_alpha": [0.012, 0.021], "taus_s": [2.0e-8, 1.5e-7],
            "source_c_lookup_zx": [2, 3], "rx_count": 4, "rx_first_m": 0.0}
    if fft:
        spec["fft_shape"] = list(fft)
    rng = np.random.default_rng(h)
    medium = np.stack((1500 + 70 * rng.standard_normal((h, w)), 1000 + 40 * rng.standard_normal((h, w))))
    return spec, DenseGeometry(spec), medium, rng.uniform(0.1, 1.0, (h, w)), rng


@pytest.mark.parametrize("h,w,pml,fft,n", [(33, 41, 6, None, 1), (70, 300, 12, None, 2), (64, 64, 4, (83, 97), 1),
                                           (300, 470, 20, (333, 501), 19), (260, 300, 24, None, 40)])
def test_dense_operator_paths(cuda, h, w, pml, fft, n):
    """The tiles and the row walk of the dense operator (its launches take the
    walk from 444 bands on) on widths around their strips, odd padded sizes and
    PML in every strip, against the FFT-evaluated oracle.  Tolerances as in the
    operator's other tests (1e-12; complex64 3e-6)."""
    from nsrno_b200.dense import DenseSystem
    from oracle import dense_ref as D
    spec, g, medium, alpha, rng = dense_case(h, w, pml, fft)
    s, o = DenseSystem(g, medium, alpha, 5.1e6, device=cuda), D.DenseSystem(D.DenseGeometry(spec), medium, alpha, 5.1e6)
    p = rng.standard_normal((n, g.H, g.W)) + 1j * rng.standard_normal((n, g.H, g.W))
    pt = torch.as_tensor(p, device=cuda)
    for adj in (False, True):
        want = [(o.adjoint if adj else o.apply)(p[k]) for k in (0, n - 1)]
        y = (s.adjoint if adj else s.apply)(pt).cpu().numpy()
        y32 = (s.adjoint if adj else s.apply)(pt.to(torch.complex64)).cpu().numpy()
        for k, ref in zip((0, n - 1), want):
            assert rel(y[k], ref) < 1e-12
            assert rel(y32[k], ref) < 3e-6


@pytest.mark.parametrize("nz,nx", [(35, 121), (57, 95), (110, 140), (85, 221), (242, 17 * 16), (1056, 38), (19, 1216),
                                   (46, 58), (61, 64)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_precondition_radices(cuda, nz, nx, adjoint):
    """Run-time transforms with every register radix (5 to 19), above it (23, 29,
    61), a single stage (19, 61) and prime last stages, against numpy's FFT; the
    tolerance of the preconditioner's other sizes (3e-6)."""
    from nsrno_b200 import precondition
    from test_gpu_operator import numpy_precondition
    rec = small_record(nz=nz, nx=nx, n_pml=4)
    med = medium_of(rec, cuda)
    x = fields(2, rec, 7).astype(np.complex64)
    y = precondition(med, torch.as_tensor(x, device=cuda), rec.frequencies, adjoint=adjoint).cpu().numpy()
    for s, f in enumerate(rec.frequencies):
        kh2 = (2 * np.pi * f / rec.c0 * rec.h) ** 2
        assert rel(y[s], numpy_precondition(x[s], nz, nx, kh2, 0.15, adjoint)) < 3e-6


@pytest.mark.parametrize("nz,nx,F", [(16, 8, 1), (67, 135, 3), (200, 264, 9)])
def test_learned_setup_tiles(cuda, nz, nx, F):
    """Gains of sizes that are no multiple of 8 nor of the network's pixel tiles,
    and more frequencies than a pixel has lanes, against the float64 oracle; the
    tolerance of the gains' other test (1e-5)."""
    from nsrno_b200.learned import LearnedPreconditioner
    from oracle import learned_ref as L
    rec = small_record(nz=nz, nx=nx, n_pml=3)
    med = medium_of(rec, cuda)
    net = LearnedPreconditioner.load(device=cuda)
    freqs = np.linspace(4.1e6, 8.8e6, F)
    gains = net.setup(med, freqs).gains.cpu().numpy()
    for k in (0, F - 1):
        ref = L.Learned(net.params.cpu().double(), rec.c, rec.rho, rec.alpha, freqs[k], rec.h, rec.c0)
        for q, want in enumerate((ref.inner, ref.outer)):
            assert rel(gains[k, q], want.detach().numpy()) < 1e-5
