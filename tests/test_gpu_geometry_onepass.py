"""One-pass 3D coefficients (iga_geometry_coefficients) against the Jacobian by
Kronecker products in numpy: degrees 1 .. 5 (band widths 2 .. 6), fewer points
than a warp, one past a warp, Gauss rules, graded knots, several segments; the
status errors.  Tolerance 1e-12 (relative max norm); the reference is formed in
extended precision from the cofactors (an FP64 inverse of J^T J is itself off by
6e-12 on the graded nets, whose displacements exceed the smallest elements)."""
import numpy as np
import pytest

from tests._problems import rel_err, rules

pytestmark = pytest.mark.gpu


def _net(rl, seed, amp=0.1):
    from igaops_b200 import unit_cube_ctrlpts

    rng = np.random.default_rng(seed)
    P = unit_cube_ctrlpts(rl)
    h = 1.0 / max(len(q.unique_kv) - 1 for q in rl)
    return P + amp * h * rng.uniform(-1.0, 1.0, P.shape)


def _reference(rl, P):
    n = [q.nbctrlpts for q in rl][::-1]
    J = np.empty((3, 3, int(np.prod([q.nbquadpts for q in rl]))), dtype=np.longdouble)
    for m in range(3):
        for j in range(3):
            t = P[m].reshape(n).astype(np.longdouble)
            for d in range(3):
                B = rl[d].basis[int(d == j)].toarray().astype(np.longdouble)
                t = np.moveaxis(np.tensordot(B, t, axes=(1, 2 - d)), 0, 2 - d)
            J[m, j] = t.reshape(-1)
    # cofactors: J^{-1} J^{-T} det J = K K^T / det J, without forming J^T J
    K = np.stack([np.cross(J[:, (i + 1) % 3], J[:, (i + 2) % 3], axis=0) for i in range(3)])
    det = np.abs(np.sum(J[:, 0] * K[0], axis=0))
    return det, np.einsum("imq,jmq->ijq", K, K) / det


def _graded(p, ne):
    from igaops_b200 import WeightedQuadrature

    inner = np.cumsum(1.5 ** np.arange(ne))
    kv = np.concatenate([np.zeros(p + 1), inner[:-1] / inner[-1], np.ones(p + 1)])
    return WeightedQuadrature(p, kv, "2")


@pytest.mark.parametrize("p", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("kind", ["small", "one_element", "ragged", "gauss", "graded", "long"])
def test_coefficients_one_pass(cuda, p, kind):
    from igaops_b200 import precompute_coefficients
    from igaops_b200.geometry import _one_pass
    from igaops_b200._device import to_device
    import torch

    if kind == "graded":
        rl = [_graded(p, 5), _graded(p, 4), _graded(p, 7)]
    elif kind == "gauss":
        rl = rules(3, p, [6, 3, 4], kind="gauss")
    else:
        rl = rules(3, p, {"small": [3, 2, 4], "one_element": 1, "ragged": [11, 3, 2],
                          "long": [2, 3, 60]}[kind])
    P = _net(rl, p)
    assert _one_pass(rl, to_device(P, torch.float64))
    out = precompute_coefficients(rl, P)
    det, C = _reference(rl, P)
    assert rel_err(out["mass"].cpu().numpy(), det) < 1e-12
    got = out["stiffness"].cpu().numpy()
    assert rel_err(got, C) < 1e-12
    assert np.array_equal(got, got.transpose(1, 0, 2))  # exactly symmetric
    assert set(precompute_coefficients(rl, P, mass=False)) == {"stiffness"}
    only = precompute_coefficients(rl, P, stiffness=False)
    assert set(only) == {"mass"} and torch.equal(only["mass"], out["mass"])


def test_singular_geometry_is_reported(cuda):
    from igaops_b200 import precompute_coefficients

    rl = rules(3, 2, 4)
    P = _net(rl, 1, amp=0.0)
    P[2] = P[1]  # a flat patch: det G = 0
    with pytest.raises(ZeroDivisionError):
        precompute_coefficients(rl, P)
    P = _net(rl, 1, amp=0.0)
    P[0, 0] = np.nan
    with pytest.raises((ZeroDivisionError, ValueError)):
        precompute_coefficients(rl, P)
