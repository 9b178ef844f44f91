"""A system's results do not depend on what runs beside it: the slots resident
at once and the slot groups they are split into regroup no sum (bitwise)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(768, 1024), (243, 729), (256, 384)], ids=lambda s: "%dx%d" % s)
def record(request, cuda):
    from nsrno_b200 import Geometry, Medium
    from nsrno_b200.media import breast_bins, breast_record
    nz, nx = request.param
    rec = breast_record(seed=3, nz=nz, nx=nx, n_pml=20, n_rx=40, rx_pitch=4, bins=breast_bins()[[0, 40]], n_angles=11)
    f, a = rec.systems()
    return Medium(Geometry.from_record(rec), rec.c, rec.rho, rec.alpha, device=cuda), f, a


SPLITS = [(22, dict(slot_groups=1)), (22, dict(slot_groups=3)), (22, dict(slot_groups=4)), (11, {}), (4, {}), (2, {}),
          (1, {})]


def check_solve(record, **shape):
    """Exactly five iterations and the FP64 residuals before and after them."""
    from nsrno_b200 import solve_batched
    med, f, a = record

    def run(n_slots, n=22, **tiles):
        r = solve_batched(med, f[:n], a[:n], tolerance=1e-30, max_iterations=5, n_slots=n_slots,
                          tiles={**shape, **tiles} or None)
        torch.cuda.synchronize()
        assert (r.iterations == 5).all()
        return r
    base = run(22)
    for n_slots, tiles in SPLITS:
        n = 22 if n_slots >= 4 else 3
        got = run(n_slots, n, **tiles)
        assert torch.equal(got.residual, base.residual[:n]), (n_slots, tiles)
        assert torch.equal(got.iq, base.iq[:n]), (n_slots, tiles)


def test_residual_sums_do_not_depend_on_the_slots(record):
    check_solve(record, stencil_rows=64)


def test_solves_do_not_depend_on_the_slots(record):
    check_solve(record)


def test_gmres_does_not_depend_on_the_slots(record):
    from nsrno_b200 import gmres_batched
    med, f, a = record
    runs = {s: gmres_batched(med, f[:11], a[:11], tolerance=1e-30, restart=6, max_iterations=6, n_slots=s,
                             return_fields=True) for s in (11, 3, 1)}
    for s in (3, 1):
        assert torch.equal(runs[s].residual, runs[11].residual)
        assert torch.equal(runs[s].fields, runs[11].fields)
