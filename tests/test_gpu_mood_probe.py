"""The redo decision of a MOOD step comes from the status word of the last
stage's own control block: a troubled step must not leave it set for the next
one, and must leave its flag in the solver's control block.  Steps after a
troubled one are compared, bit for bit, with those of a solver that has seen
nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from test_gpu_swe2d import _island_under_flow, make, moving_dam  # noqa: E402
from zoomy_b200 import _lib as L  # noqa: E402

DOMAIN = (0.0, 1.0, 0.0, 1.0)


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_a_troubled_step_leaves_the_next_alone(dtype):
    states = {"island": _island_under_flow(48), "dam": moving_dam(48, 48, DOMAIN, wet=True)}
    kw = dict(dtype=dtype, mood=True, oracle=False)

    def step(solver, name):
        Q = torch.as_tensor(np.ascontiguousarray(states[name]), device="cuda",
                            dtype=getattr(torch, dtype))
        A = solver.update_qaux(Q)
        dt = solver.compute_timestep(Q, A)
        return solver.step(dt, 0.0, Q, A)

    solver = make(48, 48, DOMAIN, states["island"], **kw)[0]
    got = [step(solver, n) for n in ("island", "dam", "island", "dam")]
    status = solver.read_ctrl().status
    assert not solver._probe.any()
    assert status & L.ZB_ST_TROUBLED    # the island's candidate has troubled cells
    for k, n in enumerate(("island", "dam")):
        fresh = step(make(48, 48, DOMAIN, states["island"], **kw)[0], n)
        assert torch.equal(got[k], fresh) and torch.equal(got[k + 2], fresh)
