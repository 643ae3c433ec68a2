"""The warp-per-tile 3D matvec kernel at the sizes where it can go wrong: tiles
cut by the grid's edge, fewer points than a tile, control ranges of one and two
8-blocks, runs of points longer and shorter than a group, windows that do not
move together (graded knots), segments without groups; every operator, both
element types, against the oracle.  Tolerances (relative max norm) as for the
other matvec tests: 1e-12 in FP64, 1e-5 in FP32."""
import numpy as np
import pytest
import torch

from oracle import mf as omf
from tests._problems import coefficients, rel_err, rules

pytestmark = pytest.mark.gpu

OPS = {"u_v": omf.mf_u_v, "gradu_gradv": omf.mf_gradu_gradv, "gradu_v": omf.mf_gradu_v,
       "u_gradv": omf.mf_u_gradv}


def _graded(p, ne):
    """Type-2 rule on knots graded towards 0 (element sizes 1 : 2 : 4 ...)."""
    from igaops_b200 import WeightedQuadrature

    inner = np.cumsum(2.0 ** np.arange(ne))
    kv = np.concatenate([np.zeros(p + 1), inner[:-1] / inner[-1], np.ones(p + 1)])
    return WeightedQuadrature(p, kv, "2")


def _case(name, p):
    if name == "one_element":       # fewer points than a tile in every direction
        return rules(3, p, 1)
    if name == "remainders":        # 1, 3 and 6 points past whole tiles (p = 2)
        return rules(3, p, [2, 5, 6])
    if name == "long":              # many groups, short faces
        return rules(3, p, [3, 2, 21])
    if name == "gauss":             # p + 1 points per element: runs cut into groups
        return rules(3, p, [4, 3, 5], kind="gauss")
    return [_graded(p, 5), _graded(p, 3), _graded(p, 6)]


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-5)])
@pytest.mark.parametrize("p", [2, 3, 4, 5])
@pytest.mark.parametrize("name", ["one_element", "remainders", "long", "gauss", "graded"])
def test_warp_kernel_edges(cuda, name, p, dtype, tol):
    from igaops_b200 import MFOperator

    rng = np.random.default_rng(100 * p + len(name))
    rl = _case(name, p)
    x = rng.standard_normal(int(np.prod([q.nbctrlpts for q in rl])))
    xd = torch.from_numpy(x).cuda().to(dtype)
    for op, oracle in OPS.items():
        for sym in ((True, False) if op == "gradu_gradv" else (True,)):
            c = coefficients(op, rl, rng, symmetric=sym)
            ref = oracle(rl, c, x)
            oper = MFOperator(rl, c, op, dtype=dtype)
            assert oper.fused
            # the chosen segment count, one segment, and more than there are groups
            for nseg in (None, 1, min(oper.plan.groups + 3, oper.plan.nq[2])):
                if nseg is not None:
                    oper.plan.set_nseg(nseg)
                assert rel_err(oper.apply(xd).cpu().numpy(), ref) < tol
            oper.plan.check_status()


def test_group_count_matches_the_device_list(cuda):
    """Groups counted on the host (segment choice) = groups listed by the library."""
    from igaops_b200.operators import FusedPlan, _GROUP_POINTS
    from igaops_b200._lib import IGA_OP_MASS

    for rl in (_case("graded", 3), _case("gauss", 5), _case("long", 2)):
        plan = FusedPlan(rl, IGA_OP_MASS, None, False, torch.float64, 1)
        row = 2 * ((plan.W + 1) // 2 * 2)  # B0 and W0, 16-byte groups
        ints = plan.step_table[plan.nq[2] * row:].view(torch.int32).cpu().numpy()
        starts = ints[1:2 + ints[0]] >> 2
        assert ints[0] == plan.groups and starts[0] == 0 and starts[-1] == plan.nq[2]
        assert np.all(np.diff(starts) >= 1) and np.all(np.diff(starts) <= _GROUP_POINTS)


def test_cta_per_tile_face_still_runs(cuda, monkeypatch):
    """A plan with the 16 x 8 face runs the CTA-per-tile kernel on its own layout."""
    from igaops_b200 import MFOperator, operators

    rng = np.random.default_rng(7)
    rl = rules(3, 3, [5, 4, 6])
    x = rng.standard_normal(int(np.prod([q.nbctrlpts for q in rl])))
    monkeypatch.setattr(operators, "FACE3", (16, 8))
    for op in ("u_v", "gradu_gradv"):
        c = coefficients(op, rl, rng)
        assert rel_err(MFOperator(rl, c, op).apply(x), OPS[op](rl, c, x)) < 1e-12
