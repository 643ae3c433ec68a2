"""Multi-patch products in several launches: patches of symmetric and of general
coefficients alternate, so that each launch has patches of non-contiguous indices and of
several band widths (degree 5 takes the wide form); and the CTA-per-tile kernel, for
plans with the 16 x 8 face."""
import numpy as np
import pytest
import torch

from oracle import mf as omf
from tests._problems import coefficients, rel_err, rules

pytestmark = pytest.mark.gpu

SPECS = [(3, 6, True), (5, 7, False), (2, 9, True), (4, 5, False), (5, 6, True), (3, 5, False)]


def _batch(specs, nseg=None):
    from igaops_b200.batch import PatchBatch

    rng = np.random.default_rng(12)
    pats = []
    for p, ne, sym in specs:
        rl = rules(3, p, ne)
        c = coefficients("gradu_gradv", rl, rng, symmetric=sym)
        pats.append((rl, torch.from_numpy(c).cuda(), np.ones((1, 3, 2), dtype=bool)))
    return pats, PatchBatch(pats, nseg=nseg)


def _refs(pats, B, x):
    out = []
    for (rl, c, _), p, xp in zip(pats, B.patches, B.split(x)):
        ref = omf.mf_gradu_gradv(rl, c.cpu().numpy(), np.asarray(xp))
        ref[p.dirichlet] = 0.0
        out.append(ref)
    return out


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-5)])
def test_launch_per_symmetry_with_skip_flags(cuda, dtype, tol):
    """A launch reads the flags of its own patches, whose indices are not its own."""
    pats, B = _batch(SPECS)
    assert len(B._mv[dtype]) == 2 and not any(g["identity"] for g in B._mv[dtype])
    x = torch.from_numpy(np.random.default_rng(9).standard_normal(B.ntot)).cuda()
    refs, xd = _refs(pats, B, x), x.to(dtype)
    for done in [()] + [(k,) for k in range(B.np)] + [(0, 3, 5)]:
        skip = torch.full((B.np,), -1, dtype=torch.int32, device="cuda")
        for k in done:
            skip[k] = k
        y = torch.empty_like(xd)
        B.matvec(xd, y, skip)
        for k, (yk, ref) in enumerate(zip(B.split(y), refs)):
            if k in done:
                assert np.all(np.asarray(yk) == 0.0), (done, k)
            else:
                assert rel_err(yk, ref) < tol, (done, k)


@pytest.mark.parametrize("p,ne,sym", [(2, (9, 4), True), (3, (6, 8), False), (5, (5, 7), True)])
def test_cta_per_tile_face(cuda, monkeypatch, p, ne, sym):
    """Plans with the 16 x 8 face, several patches in one launch."""
    from igaops_b200 import operators

    monkeypatch.setattr(operators, "FACE3", (16, 8))
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 1e-5)):
        pats, B = _batch([(p, n, sym) for n in ne], nseg=2)
        x = torch.from_numpy(np.random.default_rng(4).standard_normal(B.ntot)).cuda()
        y = torch.empty_like(x, dtype=dtype)
        B.matvec(x.to(dtype), y)
        for yk, ref in zip(B.split(y), _refs(pats, B, x)):
            assert rel_err(yk, ref) < tol
