"""The multigrid launches of a large level (a warp marching a 64-column strip)
against the float64 oracle, where they can go wrong: the smallest level that
takes them, ragged last strips and last items, sides of a few cells, every
smoothing depth, and the partial sums of z.q that the way up leaves."""
import numpy as np
import pytest
import torch

from oracle import poisson as OP
from zoomy_b200.fvm.chorin import PoissonSolver

pytestmark = pytest.mark.gpu


def depth(nx, ny):
    x = (np.arange(nx) + 0.5)[:, None] / nx
    y = (np.arange(ny) + 0.5)[None, :] / ny
    return 1.0 + 0.4 * np.sin(5 * x) * np.cos(4 * y) + 0.2 * np.sin(23 * x + 17 * y)


def rel_l2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# (nx, ny): exactly 800^2 (the first on strips) and just below it (tiles), a last
# strip of two columns, a few rows or columns only
SHAPES = [(800, 800, 2), (798, 800, 2), (804, 802, 1), (802, 892, 3), (800, 1064, 4),
          (64, 10242, 2), (10242, 64, 2), (8, 80004, 2), (80004, 8, 4)]


@pytest.mark.parametrize("nx,ny,nu", SHAPES)
def test_vcycle(nx, ny, nu):
    # one float32 V-cycle against the same in float64: the bound of the small
    # levels' test (2e-5, some 100 roundings of 6e-8 that mostly cancel)
    h = depth(nx, ny)
    dx = 1.0 / max(nx, ny)
    P = PoissonSolver(nx, ny, dx, nu=nu, coarse_sweeps=4, coarsest=4)
    P.setup(torch.as_tensor(h.reshape(-1), device="cuda"))
    H = OP.Hierarchy(*OP.face_coefficients(h), dx, coarsest=4)
    r = np.random.default_rng(nx + ny).standard_normal((nx, ny))
    z = P.vcycle(torch.as_tensor(r.reshape(-1), device="cuda", dtype=torch.float32))
    zo = OP.vcycle(H, r, nu=nu, coarse_sweeps=4)
    assert rel_l2(z.cpu().numpy().astype(np.float64).reshape(nx, ny), zo) <= 2e-5


@pytest.mark.parametrize("nx,ny", [(832, 800), (768, 1024)])
def test_solve_iterations(nx, ny):
    # a wrong z.q would cost the directions their conjugacy, and iterations
    h = depth(nx, ny)
    dx = 1.0 / nx
    b = np.random.default_rng(7).standard_normal((nx, ny))
    P = PoissonSolver(nx, ny, dx, coarse_sweeps=40, coarsest=4)   # the oracle's sweeps
    P.setup(torch.as_tensor(h.reshape(-1), device="cuda"))
    cx, cy = OP.face_coefficients(h)
    _, it_o, _ = OP.fcg(OP.Hierarchy(cx, cy, dx, coarsest=4), b, tol=1e-8, maxit=60, precond="mg")
    x, it, rel = P.solve(torch.as_tensor(b.reshape(-1), device="cuda"), tol=1e-8, maxit=60)
    res = b - OP.apply(cx, cy, x.cpu().numpy().reshape(nx, ny), dx)
    true = np.linalg.norm(res) / np.linalg.norm(b)
    assert abs(it - it_o) <= 1 and rel <= 1e-8 and true <= 1.05e-8
