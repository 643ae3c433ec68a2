"""Norms of the GMRES increment from the Gram matrix of Z: used only where they are as
good as those of the formed vectors (the bound in solvers._norms_from_gram is 1e-6)."""
import numpy as np
import pytest

from igaops_b200 import solvers


def _norms_from_gram(g, vectors):
    return solvers._norms_from_gram(g, np.sqrt(np.diag(g)), vectors)


@pytest.mark.parametrize("grade", [0, -4, -8, -12, -16])
@pytest.mark.parametrize("n", [5, 24, 400])
def test_accurate_or_refused(n, grade):
    rng = np.random.default_rng(n - grade)
    k = min(n, 24)
    V = np.linalg.qr(rng.standard_normal((n, k)))[0].T
    Z = V * np.logspace(0, grade, n)                  # rows z_i = P v_i, P graded
    if grade < -8:
        Z += rng.standard_normal(n)                   # and nearly dependent
    used = 0
    for _ in range(60):
        y = rng.standard_normal(k) * 10.0 ** rng.integers(-6, 6)
        dy = np.linalg.lstsq(Z.T, Z.T @ y * rng.random() + 1e-9 * rng.standard_normal(n), rcond=None)[0]
        for v in (y, dy, y - dy, np.linalg.svd(Z.T, full_matrices=False)[2][-1]):
            got = _norms_from_gram(Z @ Z.T, [v])
            if got is not None:
                used += 1
                exact = np.linalg.norm((Z.T.astype(np.longdouble) @ v).astype(float))
                assert abs(got[0] - exact) <= 1e-6 * exact
    assert used or grade < -8


def test_cancelled_form_is_refused():
    """A form that rounding makes zero or negative is not a norm of zero."""
    z = np.ones(7)
    Z = np.stack([z, z * (1 + 1e-12)])
    assert _norms_from_gram(Z @ Z.T, [np.array([1.0, -1.0])]) is None
    assert _norms_from_gram(np.array([[1.0, 1.0], [1.0, 1.0 - 1e-16]]), [np.array([1.0, -1.0])]) is None
    assert _norms_from_gram(Z @ Z.T, [np.zeros(2)]) is None  # y = 0: the formed vectors decide
