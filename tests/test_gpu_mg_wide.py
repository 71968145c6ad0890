"""The pressure solve on a level so wide that its strips exceed the slots for partial sums of
z.q (more than 851,968 columns at two sweeps): the direction's scalar then comes from a pass
of its own, and the solve converges as on a narrower level of the same height."""
import numpy as np
import pytest
import torch

from oracle import poisson as OP
from zoomy_b200.fvm.chorin import PoissonSolver

pytestmark = pytest.mark.gpu


def solve(nx, ny):
    x = (np.arange(nx) + 0.5)[:, None] / nx
    y = (np.arange(ny) + 0.5)[None, :]
    h = 1.0 + 0.4 * np.sin(5 * x) * np.cos(0.3 * y) + 0.2 * np.sin(17 * x + 0.7 * y)
    b = np.random.default_rng(5).standard_normal((nx, ny))
    P = PoissonSolver(nx, ny, 1.0 / nx)
    P.setup(torch.as_tensor(h.reshape(-1), device="cuda"))
    p, it, rel = P.solve(torch.as_tensor(b.reshape(-1), device="cuda"), tol=1e-8, maxit=60)
    res = b - OP.apply(*OP.face_coefficients(h), p.cpu().numpy().reshape(nx, ny), 1.0 / nx)
    return it, rel, np.linalg.norm(res) / np.linalg.norm(b)


def test_more_strips_than_partial_sums():
    it, rel, true = solve(8, 900000)
    # the same equations on a tenth of the columns, whose strips fit the slots
    it_narrow, _, _ = solve(8, 90000)
    assert rel <= 1e-8 and true <= 1.05e-8
    assert abs(it - it_narrow) <= 1
