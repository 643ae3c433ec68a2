"""GMRES with preconditioners that leave Z = P V badly scaled: the increment criterion
must not end the solve on a rounding of the Gram matrix of Z (it did with a residual of
0.3). Against the oracle's GMRES, which forms the difference."""
import numpy as np
import pytest
import torch

from oracle import krylov as okr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grade,tol", [(24, -10, 1e-6), (48, -10, 1e-6), (24, -6, 1e-8),
                                         (24, 0, 1e-10)])
def test_graded_preconditioner(cuda, n, grade, tol):
    from igaops_b200.solvers import LinearSolver

    rng = np.random.default_rng(1)
    A = np.eye(n) + 0.3 * rng.standard_normal((n, n)) / np.sqrt(n)
    p = np.logspace(0, grade, n)
    b = rng.standard_normal(n)
    x, res, ok, its = okr.gmres(lambda v: A @ v, b, lambda v: p * v, tol=tol, maxiters=n + 6)
    assert ok and np.linalg.norm(b - A @ x) < 1e-5 * np.linalg.norm(b)
    Ad, pd = torch.from_numpy(A).cuda(), torch.from_numpy(p).cuda()
    out = LinearSolver(tol, n + 6, linear_type="gmres", verbose=False).solve(
        lambda v: Ad @ v, b, lambda v: pd * v)
    assert out.success
    assert abs(len(out.residual) - 1 - its) <= 1, (len(out.residual) - 1, its)
    assert np.linalg.norm(b - A @ out.solution) < 1e-5 * np.linalg.norm(b)
