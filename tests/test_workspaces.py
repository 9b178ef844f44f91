"""Workspace sizes (no GPU; they are host functions of the library)."""
import ctypes

import pytest


@pytest.mark.parametrize("nz,nx,slots,restart", [(768, 1024, 11, 8), (256, 256, 4, 32), (512, 768, 1, 4)])
def test_gmres_workspace_holds_its_vectors_and_little_more(nz, nx, slots, restart):
    """Per slot: the basis (restart + 1 planes), w, the transform's work field and
    the residual in complex64, two complex128 iterates; the rest is less than
    half a plane."""
    from nsrno_b200 import _lib
    try:
        lib = _lib.load()
    except RuntimeError:
        pytest.skip("the library has not been built")
    grid = _lib.NsrGrid()
    grid.nz, grid.nx, grid.n_pml, grid.face, grid.h, grid.c0, grid.rho0 = nz, nx, 20, 4, 1e-4, 1540.0, 1000.0
    grid.pml_strength, grid.alpha_power, grid.aperture_half_width = 3.0, 1.1, 0.0
    size = lib.nsr_gmres_workspace_size(ctypes.byref(grid), slots, restart)
    plane = 8 * nz * nx * slots
    vectors = plane * (restart + 1 + 3) + 4 * plane
    assert vectors < size < vectors + plane // 2
