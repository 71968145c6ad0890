"""The triangle step's workspace: laid out from its first 16-byte boundary, so a
workspace of any element alignment gives the same bits."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import zoomy_b200 as zb  # noqa: E402
from zoomy_b200 import _lib as L  # noqa: E402
from zoomy_b200.fvm.solver import HyperbolicSolver  # noqa: E402
from zoomy_b200.trimesh import TriangleMesh  # noqa: E402


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n_side", [3, 12])
def test_workspace_alignment_does_not_change_the_step(n_side, dtype):
    mesh = TriangleMesh.create(n_side, seed=1)
    xc = mesh.cell_centers()
    h = np.where(xc[0] < 0.5, 2.0, 1.0)
    Q0 = np.stack([0.1 * xc[1], h, 0.1 * h, -0.2 * h])
    tags = ("left", "right", "bottom", "top")
    model = zb.ShallowWater2D(boundary_conditions={t: "wall" for t in tags},
                              initial_conditions=Q0)
    nsm = zb.NumericalSystemModel.from_system_model(model, zb.ReconstructionSpec(2, "minmod"),
                                                    "hll_hr")
    s = HyperbolicSolver(time_end=math.inf, compute_dt=zb.timestepping.adaptive(0.4, 2),
                         reconstruction_variables="eta", free_surface_h_index=1, dtype=dtype)
    Q, _ = s.setup_simulation(mesh, nsm)
    es = 4 if dtype == "float32" else 8
    nb = s._ws_bytes
    buf = torch.zeros(nb + 64, dtype=torch.uint8, device="cuda")
    outs = []
    for off in (0, es, 3 * es if es == 4 else es):
        q = Q.clone()
        s.init_march(q)
        for k in range(2):
            rc = s.be.step(L.ptr(q), C.c_void_p(buf.data_ptr() + off), C.c_size_t(nb),
                           L.ptr(s._ctrl), k, s._s())
            assert rc == L.ZB_OK
        assert not torch.equal(q, Q) and bool(torch.isfinite(q).all())
        outs.append(q)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
