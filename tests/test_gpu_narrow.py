"""Grids without a middle strip (fewer than 58 columns) above the uniform list's limit of 3552
strip rows: one list of items of the general body, ragged last items, against the float64
oracle.  Tolerances as in test_gpu_strip_body.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import swe as OS  # noqa: E402
from test_gpu_strip_body import SCHEMES, SIDES, case  # noqa: E402
from test_gpu_swe2d import rel_err  # noqa: E402


@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 2e-5)])
@pytest.mark.parametrize("bc", [SIDES[0], SIDES[2], SIDES[4]], ids=str)
@pytest.mark.parametrize("nx,ny", [(3553, 28), (1801, 57), (9001, 30)])
def test_step_and_stage(nx, ny, bc, dtype, tol):
    Q0, (solver, Q, Qaux, om, sch, params) = case(nx, ny, bc, SCHEMES[0], dtype)
    dt = float(np.float32(0.5 * OS.compute_dt(om, Q0, params, sch)))
    ref = OS.step(om, Q0, dt, params, sch)
    got = solver.step(dt, 0.0, Q, Qaux)
    assert rel_err(got.double().cpu().numpy(), ref).max() <= tol
    solver.cfg.dt_max = dt
    solver.init_march(Q)
    solver.launch_steps(Q, 1)
    c = solver.read_ctrl()
    assert c.steps == 1 and c.dt == dt
    assert rel_err(Q.double().cpu().numpy(), ref).max() <= tol
