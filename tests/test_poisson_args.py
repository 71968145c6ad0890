"""What the pressure solve's entry points refuse before they touch the device: a V-cycle
whose levels would take no smoothing sweep (nu = 0).  Configurations in which no level is
smoothed stay accepted."""
import ctypes as C

import pytest
import torch

from zoomy_b200 import _lib as L

# a call that is not refused would launch on addresses that are no device memory
pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="host checks only")


def cfg(nx, ny, nu, coarsest=4):
    return L.ZbPoissonCfg(nx, ny, 1.0 / nx, 0.1, 2.0, nu, 8, coarsest)


def codes(c, precond):
    """Return codes of the four entry points that run a preconditioner."""
    lib = L.load()
    buf = C.addressof(C.create_string_buffer(4096))
    p = C.c_void_p(buf)
    smo = L.ZbSmoother()
    sp = C.byref(smo) if precond >= 2 else None
    g = C.c_void_p()
    return [lib.zb_poisson_vcycle(C.byref(c), p, p, p, precond, sp, None),
            lib.zb_fcg_start(C.byref(c), p, p, p, precond, sp, None),
            lib.zb_fcg_iterate(C.byref(c), p, p, precond, sp, None),
            lib.zb_fcg_graph_create(C.byref(c), p, p, p, precond, sp, 1e-8, 10, C.byref(g), None)]


SMOOTHED = [(nx, ny, precond) for nx, ny in [(8, 8), (32, 32), (64, 64), (1024, 1024)]
            for precond in (1, 2, 3)] + [(8, 80004, 1), (8, 80004, 2)]


@pytest.mark.parametrize("nx,ny,precond", SMOOTHED)
def test_unsmoothed_levels_are_refused(nx, ny, precond):
    assert codes(cfg(nx, ny, 0), precond) == [L.ZB_E_UNSUPPORTED] * 4


@pytest.mark.parametrize("nx,ny,coarsest,precond",
                         [(1024, 1024, 4, 0), (4, 4, 4, 1), (33, 64, 4, 1), (64, 64, 32, 3),
                          (8, 80004, 4, 3)])
def test_configurations_without_smoothed_levels_are_accepted(nx, ny, coarsest, precond):
    c = cfg(nx, ny, 0, coarsest)
    assert L.load().zb_poisson_workspace_bytes(C.byref(c)) > 0
    assert L.ZB_E_UNSUPPORTED not in codes(c, precond)
