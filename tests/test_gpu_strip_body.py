"""The strip kernel's general (boundary) body and its item lists at the grid
sizes where they can go wrong, against the float64 oracle.

Tolerance: float64 relative L-infinity <= 1e-12 per state row and step, the
bound of the other Cartesian parity tests (a stage is a few hundred operations
on values of order one; the corner cells' closed form and the class weights it
restates agree to a few ulp).  float32 <= 2e-5: one step of the float32
arithmetic (2^-24 relative per operation, about 300 of them per cell) from the
same float32-rounded state and dt.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import swe as OS  # noqa: E402
from test_gpu_swe2d import make, moving_dam, rel_err  # noqa: E402
from zoomy_b200 import _lib as L  # noqa: E402

# 3 cells: every cell touches a boundary; 28 / 29 / 30 / 58 columns: the last
# strip one column wide, no middle strip, the first middle strip; 720 x 140:
# both bodies in one launch (the smaller ones take the general body alone)
SIZES = [(3, 3), (3, 40), (40, 3), (4, 28), (9, 29), (33, 30), (64, 58), (57, 85)]
SIDES = ["wall", "extrapolation", "periodic", ("periodic", "periodic", "wall", "extrapolation"),
         ("extrapolation", "wall", "periodic", "periodic")]
SCHEMES = [
    dict(recon="eta", riemann="hll_hr", eps_wet=1e-6),
    dict(recon="eta", riemann="rusanov_hr", limiter="venkatakrishnan", manning=0.03),
    dict(recon="conservative", riemann="hll_hr"),
]


def case(nx, ny, bc, scheme, dtype):
    domain = (0.0, 0.02 * nx, 0.0, 0.03 * ny)
    Q0 = moving_dam(nx, ny, domain, wet=scheme["recon"] == "conservative")
    Q0 = Q0.astype(np.float32).astype(np.float64)
    return Q0, make(nx, ny, domain, Q0, bc=bc, dtype=dtype, **scheme)


@pytest.mark.parametrize("scheme", SCHEMES, ids=lambda s: "-".join(str(v) for v in s.values()))
@pytest.mark.parametrize("bc", SIDES, ids=str)
@pytest.mark.parametrize("nx,ny", SIZES)
def test_step_and_stage_match_oracle(nx, ny, bc, scheme):
    Q0, (solver, Q, Qaux, om, sch, params) = case(nx, ny, bc, scheme, "float64")
    dt = 0.5 * OS.compute_dt(om, Q0, params, sch)
    ref = OS.step(om, Q0, dt, params, sch)
    # the generic stages
    got = solver.step(dt, 0.0, Q, Qaux).cpu().numpy()
    assert rel_err(got, ref).max() <= 1e-12
    # the fused step
    solver.cfg.dt_max = dt
    solver.init_march(Q)
    solver.launch_steps(Q, 1)
    assert solver.read_ctrl().dt == dt
    assert rel_err(Q.cpu().numpy(), ref).max() <= 1e-12


@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 2e-5)])
@pytest.mark.parametrize("bc", [SIDES[0], SIDES[2], SIDES[4]], ids=str)
@pytest.mark.parametrize("nx,ny", [(57, 85), (720, 140)])
def test_both_bodies_in_one_launch(nx, ny, bc, dtype, tol):
    Q0, (solver, Q, Qaux, om, sch, params) = case(nx, ny, bc, SCHEMES[0], dtype)
    dt = float(np.float32(0.5 * OS.compute_dt(om, Q0, params, sch)))
    ref = OS.step(om, Q0, dt, params, sch)
    solver.cfg.dt_max = dt
    solver.init_march(Q)
    solver.launch_steps(Q, 1)
    c = solver.read_ctrl()
    assert c.steps == 1 and c.dt == dt
    assert rel_err(Q.double().cpu().numpy(), ref).max() <= tol


@pytest.mark.parametrize("bc", [SIDES[0], SIDES[3]], ids=str)
@pytest.mark.parametrize("nx,ny", [(9, 29), (57, 85), (720, 140)])
def test_stage_mask_and_troubled_output(nx, ny, bc):
    """The generic stage's first-order mask against the oracle's, and its
    troubled mask on a state with negative and non-finite cells."""
    Q0, (solver, Q, Qaux, om, sch, params) = case(nx, ny, bc, SCHEMES[0], "float64")
    rng = np.random.default_rng(1)
    mask = rng.uniform(size=nx * ny) < 0.3
    dt = 0.3 * OS.compute_dt(om, Q0, params, sch)
    kind = OS.bc_kinds(om, sch)
    ref = Q0 + dt * OS.flux_operator(om, Q0, sch, params, kind, mask)
    out = torch.empty_like(Q)
    out[0].copy_(Q[0])
    fo = torch.as_tensor(mask.astype(np.uint8), device=Q.device)
    tr = torch.full((nx * ny,), 7, dtype=torch.uint8, device=Q.device)
    solver._stage(solver.cfg, Q, None, out, 0.0, 1.0, dt, fo=fo, tr=tr)
    assert rel_err(out.cpu().numpy(), ref).max() <= 1e-12
    assert np.array_equal(tr.cpu().numpy().astype(bool), OS.troubled_cells(ref))
    # a non-finite cell: its own entry is flagged, and the status word
    Qbad = Q.clone()
    k = (nx // 2) * ny + ny // 2
    Qbad[2, k] = float("nan")
    solver._stage(solver.cfg, Qbad, None, out, 0.0, 1.0, dt, tr=tr)
    assert int(tr[k]) == 1 and solver.read_ctrl().status & L.ZB_ST_TROUBLED
