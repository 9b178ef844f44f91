"""Edges of the C entry points: buffers in place, refused calls, odd alignments,
values outside the physical range."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel
from test_gpu_operator import medium_of, small_record

pytestmark = pytest.mark.gpu


def ptr(t, offset=0):
    return ctypes.c_void_p(t.data_ptr() + offset)


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("nx", [256, 384])
def test_workspaces_aligned_to_eight_bytes(cuda, nx):
    """Row transforms of the specialised widths move 16 bytes at a time; a
    workspace that is aligned to its 8-byte elements only gives the same result
    by other kernels (two transforms within 3e-6 of the exact one: 6e-6)."""
    from nsrno_b200 import _lib
    from nsrno_b200.dense import DenseSystem
    from nsrno_b200.learned import N_PARAMS, LearnedPreconditioner
    from test_gpu_tiles import dense_case
    rec = small_record(nz=48, nx=nx)
    med = medium_of(rec, cuda)
    net = LearnedPreconditioner.load(device=cuda)
    setup = net.setup(med, rec.frequencies)
    lib = _lib.load()
    grid, S = ctypes.byref(med._grid), 2
    f = torch.as_tensor(rec.frequencies, device=cuda)
    x = torch.randn((S, rec.nz, nx), dtype=torch.complex64, device=cuda)
    x2 = torch.randn_like(x)
    struct = setup.struct(torch.arange(S, dtype=torch.int32, device=cuda))
    size = lib.nsr_precondition_workspace_size(grid, S)
    spec_size = lib.nsr_learned_spectral_workspace_size(grid, S)
    _, g, medium, alpha, _ = dense_case(24, 40, 4, (48, nx))
    dense = DenseSystem(g, medium, alpha, 5.1e6, device=cuda)
    p = torch.randn((S, g.H, g.W), dtype=torch.complex64, device=cuda)
    dense_size = lib.nsr_dense_precondition_workspace_size(ctypes.byref(g.struct), S)
    ws = torch.empty(max(size, spec_size, dense_size) + 16, dtype=torch.uint8, device=cuda)

    def results(off):
        y, ly, dy = torch.empty_like(x), torch.empty_like(x), torch.empty_like(p)
        dp = torch.zeros(N_PARAMS, device=cuda)
        for adj in (0, 1):
            assert lib.nsr_precondition(grid, ptr(f), S, 0.15, adj, ptr(x), ptr(y), ptr(ws, off), size, stream()) == 0
            assert lib.nsr_learned_precondition(grid, ctypes.byref(struct), ptr(f), S, adj, ptr(x), ptr(ly),
                                                ptr(ws, off), size, stream()) == 0
            assert lib.nsr_dense_precondition(ctypes.byref(g.struct), float((dense.k0 * g.dx) ** 2), 0.15, S, adj,
                                              ptr(p), ptr(dy), ptr(ws, off), dense_size, stream()) == 0
            yield from (v.cpu().numpy().copy() for v in (y, ly, dy))
        assert lib.nsr_learned_spectral_backward(grid, ptr(net.params), ptr(f), S, ptr(x), ptr(x2), ptr(dp),
                                                 ptr(ws, off), spec_size, stream()) == 0
        yield dp.cpu().numpy()
    for want, got in zip(results(0), results(8)):
        assert np.abs(want).max() > 0
        assert rel(got, want) < 6e-6


@pytest.mark.parametrize("bad", [-1, 2, 1 << 30])
def test_refused_gain_index_leaves_the_output_alone(cuda, bad):
    from nsrno_b200 import _lib
    from nsrno_b200.learned import LearnedPreconditioner
    rec = small_record(nz=64, nx=96)
    med = medium_of(rec, cuda)
    setup = LearnedPreconditioner.load(device=cuda).setup(med, rec.frequencies)
    lib = _lib.load()
    S = 3
    index = torch.tensor([0, 1, bad], dtype=torch.int32, device=cuda)
    f = torch.as_tensor(rec.frequencies[[0, 1, 1]], device=cuda)
    x = torch.randn((S, rec.nz, rec.nx), dtype=torch.complex64, device=cuda)
    y = torch.full_like(x, 7.0)
    size = lib.nsr_precondition_workspace_size(ctypes.byref(med._grid), S)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda)
    struct = setup.struct(index)
    code = lib.nsr_learned_precondition(ctypes.byref(med._grid), ctypes.byref(struct), ptr(f), S, 0, ptr(x), ptr(y),
                                        ptr(ws), size, stream())
    torch.cuda.synchronize()
    assert code != 0
    assert (y == 7.0).all()


@pytest.mark.parametrize("c_bad,rho_bad,alpha_bad", [
    (-1500.0, None, None), (None, -1000.0, None), (0.0, None, None), (None, np.inf, None), (None, None, np.inf),
    (None, None, -1.0), (None, None, -1.0 + 2.0 ** -24), (None, None, -2.0)])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_context_of_values_outside_the_physical_range(cuda, c_bad, rho_bad, alpha_bad, count):
    """The pooled context is the mean of the nodes' logarithms also where a
    medium has values that no tissue has, one to four of them in a column:
    negative ones give NaN, zeros and infinities what their logarithms give."""
    from nsrno_b200 import _lib
    from nsrno_b200.learned import LearnedPreconditioner
    rec = small_record(nz=24, nx=40, n_pml=3)
    med = medium_of(rec, cuda)
    net = LearnedPreconditioner.load(device=cuda)
    planes = [np.array(v, np.float32) for v in (rec.c, rec.rho, rec.alpha)]
    for v, value in zip(planes, (c_bad, rho_bad, alpha_bad)):
        if value is not None:
            v[8:8 + count, 19] = value
    lib = _lib.load()
    f = torch.tensor([2.3e6], dtype=torch.float64, device=cuda)
    state = torch.zeros(lib.nsr_learned_state_bytes(ctypes.byref(med._grid), 1), dtype=torch.uint8, device=cuda)
    dev = [torch.as_tensor(v, device=cuda) for v in planes]
    assert lib.nsr_learned_setup(ctypes.byref(med._grid), *[ptr(v) for v in dev], ptr(f), 1, ptr(net.params),
                                 ptr(state), None, stream()) == 0
    got = state[:4 * 3 * 15].view(torch.float32).reshape(3, 3, 5).cpu().numpy()
    with np.errstate(all="ignore"):
        c, rho, alpha = (v.astype(np.float64) for v in planes)
        logs = np.stack((np.log(c / 1540) / 0.06, np.log(rho / 1000) / 0.08, np.log1p(alpha)))
        want = logs.reshape(3, 3, 8, 5, 8).mean(axis=(2, 4))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    ok = np.isfinite(want)
    # rounding of the mean to float: 6e-8 of the largest term
    assert np.abs(got[ok] - want[ok]).max() < 1e-6 * np.abs(want[ok]).max()


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("h,w,pml,n", [(70, 300, 12, 2), (260, 300, 24, 40), (130, 150, 12, 19)])
def test_dense_apply_in_place(cuda, h, w, pml, n, dtype):
    """y = x is the same buffer: the result of separate buffers, bit for bit (row
    walk and tiles)."""
    from nsrno_b200 import _lib
    from nsrno_b200.dense import DenseSystem
    from test_gpu_tiles import dense_case
    _, g, medium, alpha, rng = dense_case(h, w, pml)
    s = DenseSystem(g, medium, alpha, 5.1e6, device=cuda)
    p = torch.as_tensor(rng.standard_normal((n, g.H, g.W)) + 1j * rng.standard_normal((n, g.H, g.W)),
                        device=cuda).to(dtype)
    lib = _lib.load()
    prec = int(dtype == torch.complex128)
    size = lib.nsr_dense_workspace_size(ctypes.byref(g.struct), n, prec)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda)
    for adj in (0, 1):
        want = (s.adjoint if adj else s.apply)(p)
        y = p.clone()
        assert lib.nsr_dense_apply(ctypes.byref(g.struct), ptr(s.coef), s.scal.real, s.scal.imag, n, adj, prec,
                                   ptr(y), ptr(y), ptr(ws), size, stream()) == 0
        assert torch.equal(y, want)
