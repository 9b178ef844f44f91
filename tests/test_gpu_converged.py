"""A batch whose systems all start converged runs no round of the device loop."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_converged_batch_runs_no_round(cuda):
    from nsrno_b200 import Geometry, Medium, solve_batched
    from nsrno_b200.media import breast_record
    from nsrno_b200.solver import solve_progress
    rec = breast_record()
    med = Medium(Geometry.from_record(rec), rec.c, rec.rho, rec.alpha, device=cuda)
    f, a = rec.systems()
    r = solve_batched(med, f[:22], a[:22], tolerance=2.0, n_slots=22)
    torch.cuda.synchronize()
    assert r.reasons() == ["converged"] * 22 and int(r.iterations.sum()) == 0
    done, rounds, error, _ = solve_progress(r)
    assert (done, rounds, error) == (22, 0, 0)
