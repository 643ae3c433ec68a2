"""The warp-per-tile 2D matvec kernel at the sizes where it can go wrong: fewer
points than a tile, one past a tile, output ranges above 32, runs cut into
groups, windows that move apart (graded knots), segments without groups, several
columns; every operator, both element types, against the oracle (1e-12 FP64,
1e-5 FP32, relative max norm, as for the other matvec tests)."""
import numpy as np
import pytest
import torch

from oracle import mf as omf
from tests._problems import coefficients, rel_err, rules

pytestmark = pytest.mark.gpu

OPS = {"u_v": omf.mf_u_v, "gradu_gradv": omf.mf_gradu_gradv, "gradu_v": omf.mf_gradu_v,
       "u_gradv": omf.mf_u_gradv}


def _graded(p, ne):
    from igaops_b200 import WeightedQuadrature

    inner = np.cumsum(2.0 ** np.arange(ne))
    kv = np.concatenate([np.zeros(p + 1), inner[:-1] / inner[-1], np.ones(p + 1)])
    return WeightedQuadrature(p, kv, "2")


def _case(name, p):
    if name == "one_element":
        return rules(2, p, 1)
    if name == "past_a_tile":    # 33 .. points in direction 1 for p = 2 (3 ne + 2 p - 1)
        return rules(2, p, [10, 4])
    if name == "long":
        return rules(2, p, [25, 40])
    if name == "gauss":
        return rules(2, p, [9, 7], kind="gauss")
    return [_graded(p, 6), _graded(p, 8)]


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-5)])
@pytest.mark.parametrize("p", [2, 3, 4, 5])
@pytest.mark.parametrize("name", ["one_element", "past_a_tile", "long", "gauss", "graded"])
def test_warp_kernel_2d_edges(cuda, name, p, dtype, tol):
    from igaops_b200 import MFOperator

    rng = np.random.default_rng(10 * p + len(name))
    rl = _case(name, p)
    x = rng.standard_normal((int(np.prod([q.nbctrlpts for q in rl])), 2))
    xd = torch.from_numpy(x).cuda().to(dtype)
    for op, oracle in OPS.items():
        for sym in ((True, False) if op == "gradu_gradv" else (True,)):
            c = coefficients(op, rl, rng, symmetric=sym)
            ref = np.stack([oracle(rl, c, x[:, k]) for k in range(2)], axis=1)
            oper = MFOperator(rl, c, op, dtype=dtype)
            assert oper.fused and oper.plan.resident >= 1
            for nseg in (None, 1, min(oper.plan.groups + 2, oper.plan.nq[1])):
                if nseg is not None:
                    oper.plan.set_nseg(nseg)
                assert rel_err(oper.apply(xd).cpu().numpy(), ref) < tol
            oper.plan.check_status()


def test_cta_per_tile_face_2d_still_runs(cuda, monkeypatch):
    from igaops_b200 import MFOperator, operators

    rng = np.random.default_rng(8)
    rl = rules(2, 3, [50, 9])
    x = rng.standard_normal(int(np.prod([q.nbctrlpts for q in rl])))
    monkeypatch.setattr(operators, "FACE2", (128,))
    for op in ("u_v", "gradu_gradv"):
        c = coefficients(op, rl, rng)
        assert rel_err(MFOperator(rl, c, op).apply(x), OPS[op](rl, c, x)) < 1e-12


@pytest.mark.parametrize("ndim,op", [(2, "u_v"), (2, "gradu_gradv"), (3, "u_v"), (3, "gradu_v")])
def test_strip_of_more_points_than_a_grid_axis(cuda, ndim, op):
    """A long strip: more than 65535 points in the streamed direction (one axis of a
    launch grid), few in the others."""
    from igaops_b200 import MFOperator

    rng = np.random.default_rng(5)
    rl = rules(ndim, 2, [2] * (ndim - 1) + [21850], kind="gauss")
    assert rl[-1].nbquadpts > 65535
    c = coefficients(op, rl, rng)
    x = rng.standard_normal(int(np.prod([q.nbctrlpts for q in rl])))
    oper = MFOperator(rl, c, op)
    assert oper.fused
    assert rel_err(oper.apply(x), OPS[op](rl, c, x)) < 1e-12
    oper.plan.check_status()
