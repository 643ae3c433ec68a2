"""Which outputs an infinity or NaN in x or in the coefficients may reach. In 2D, the
control windows and test bands of the points it enters, as wide as the plan pads them. In
3D, the tensor-core products run over whole tiles of 8 x 8 points, zero weights included:
the outputs of the tiles whose control ranges (points, for a coefficient) hold it, and the
windows of the streamed direction. What it must reach: the outputs that the oracle's
operator couples to it. All others have the oracle's values (1e-12 FP64, 1e-5 FP32,
relative max norm, as for the other matvec tests)."""
import numpy as np
import pytest
import torch

from igaops_b200.bands import rule_bands
from oracle import mf as omf
from tests._problems import coefficients, rel_err, rules

pytestmark = pytest.mark.gpu

OPS = {"u_v": omf.mf_u_v, "gradu_gradv": omf.mf_gradu_gradv, "gradu_v": omf.mf_gradu_v,
       "u_gradv": omf.mf_u_gradv}


def _reach(q, W, RW, tile, last):
    """(units that a control point enters, outputs that a unit enters, unit of a point):
    a unit is a point, or a tile of `tile` points."""
    rb = rule_bands(q)
    c, p = np.arange(rb.n), np.arange(rb.nq)
    ts, ws = rb.trial[0], rb.testT[0]
    if tile > 1:
        lo = np.arange(0, rb.nq, tile)
        hi = np.minimum(lo + tile, rb.nq) - 1
        units = (c[None, :] >= ts[lo][:, None]) & (c[None, :] < ts[hi][:, None] + W)
        outputs = (c[:, None] >= ws[lo][None, :]) & (c[:, None] < ws[hi][None, :] + W)
        return units.astype(float), outputs.astype(float), p // tile
    units = (c[None, :] >= ts[:, None]) & (c[None, :] < ts[:, None] + W)
    if last:
        outputs = (c[:, None] >= ws[None, :]) & (c[:, None] < ws[None, :] + W)
    else:
        rs = rb.testR[0][:, None]
        outputs = (p[None, :] >= rs) & (p[None, :] < rs + RW)
    return units.astype(float), outputs.astype(float), p


def _kron(vectors):  # direction 1 fastest
    out = np.ones(1)
    for v in vectors:
        out = np.outer(v, out).reshape(-1)
    return out


def _check(oper, y, may, must, clean, tol):
    bad = ~np.isfinite(y)
    assert not np.any(bad & ~may), f"{np.sum(bad & ~may)} outputs out of reach are not finite"
    assert not np.any(must & ~bad), f"{np.sum(must & ~bad)} outputs missed it"
    assert rel_err(np.where(bad, 0.0, y), np.where(bad, 0.0, clean)) < tol
    oper.plan.check_status()


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-5)])
@pytest.mark.parametrize("p,ne,kind", [(2, [11, 9, 10], "wq2"), (3, [9, 10, 8], "gauss"),
                                       (5, [9, 8, 11], "wq2"), (4, [1, 8, 9], "wq2"),
                                       (3, [30, 17], "wq2"), (5, [24, 12], "gauss")])
def test_nonfinite_values_stay_in_reach(cuda, p, ne, kind, dtype, tol):
    from igaops_b200 import MFOperator

    rng = np.random.default_rng(10 * p + len(ne))
    rl = rules(len(ne), p, ne, kind=kind)
    n, nq = [q.nbctrlpts for q in rl], [q.nbquadpts for q in rl]
    N, NQ = int(np.prod(n)), int(np.prod(nq))
    x = rng.uniform(0.5, 1.5, N)
    for op, oracle in OPS.items():
        if op == "u_gradv" and p != 3:
            continue
        c = coefficients(op, rl, rng)
        oper = MFOperator(rl, c, op, dtype=dtype)
        assert oper.fused
        W, RW = oper.plan.W, oper.plan.RW
        last = len(rl) - 1
        reach = [_reach(q, W, RW, 8 if len(rl) == 3 and d < last else 1, d == last)
                 for d, q in enumerate(rl)]
        for at, value in ((0, np.nan), (N - 1, np.inf), (int(rng.integers(N)), np.inf),
                          (int(rng.integers(N)), np.nan), (int(rng.integers(N)), -np.inf)):
            idx = np.unravel_index(at, n, order="F")
            may = _kron([o @ t[:, i] for (t, o, _), i in zip(reach, idx)]) > 0
            unit = np.zeros(N)
            unit[at] = 1.0
            unit = np.abs(oracle(rl, c, unit))
            xb, xc = x.copy(), x.copy()
            xb[at], xc[at] = value, 0.0
            y = oper.apply(torch.from_numpy(xb).cuda().to(dtype)).double().cpu().numpy()
            _check(oper, y, may, unit > 1e-6 * unit.max(), oracle(rl, c, xc), tol)
        # one coefficient of one quadrature point
        for at in (NQ - 1, int(rng.integers(NQ))):
            idx = np.unravel_index(at, nq, order="F")
            may = _kron([o[:, u[i]] for (t, o, u), i in zip(reach, idx)]) > 0
            cb, cc, only = c.copy(), c.copy(), np.zeros_like(c)
            only[..., at] = c[..., at]
            cc[..., at] = 0.0
            cb[..., at] = np.nan
            unit = np.abs(oracle(rl, only, x))
            bad = MFOperator(rl, cb, op, dtype=dtype, symmetric=oper.symmetric)
            y = bad.apply(torch.from_numpy(x).cuda().to(dtype)).double().cpu().numpy()
            _check(bad, y, may, unit > 1e-6 * unit.max(), oracle(rl, cc, x), tol)
