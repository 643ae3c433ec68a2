"""Space-time FD apply with the time part in one kernel, at its edges: time extents
around the k-steps, the 8-row blocks, the warp and the shared-memory limit (104 /
105, the last on the separate launches), spatial sizes cut by the 16-column tile,
one to three space directions, both precisions, against the oracle.  Tolerances as
for the other space-time tests (1e-11 FP64, 1e-5 FP32, relative max norm)."""
import numpy as np
import pytest
import torch

from oracle import fd as ofd
from tests._problems import rel_err, rules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sdim,ne,mt", [(2, 3, 2), (2, 5, 3), (1, 16, 4), (2, 4, 5), (3, 2, 8),
                                        (2, 6, 9), (1, 15, 31), (2, 4, 32), (2, 3, 33),
                                        (1, 9, 104), (1, 9, 105)])
def test_sptime_time_kernel_edges(cuda, sdim, ne, mt):
    from igaops_b200.fastdiag import SingleFD, rewrite_quadrature

    p = 2 if mt > 2 else 1  # mt = elements + p - 1
    space = rules(sdim, 2, ne)
    qt = rules(1, p, mt - p + 1)[0]
    assert qt.nbctrlpts - 1 == mt
    table = np.ones((1, sdim, 2), dtype=bool)
    table[0, -1, 0] = False
    fd = SingleFD("spacetime")
    fd.compute_space_eigendecomposition(space, table)
    fd.compute_time_schurdecomposition(qt)
    fd.update_space_eigenvalues(scalar_coefs=(0.3, 1.0))
    fd.add_scalar_space_time_correctors(advection_corrector=[0.8])
    ref = ofd.sptime_setup(rewrite_quadrature(space), table, rewrite_quadrature([qt])[0],
                           scalar_coefs=(0.3, 1.0), adv_corr=0.8)
    x = np.random.default_rng(mt).standard_normal(
        int(np.prod([q.nbctrlpts for q in space])) * qt.nbctrlpts)
    assert rel_err(fd.apply(x), ofd.sptime_apply(ref, x)) < 1e-11
    assert rel_err(fd.apply_transpose(x), ofd.sptime_apply(ref, x, transpose=True)) < 1e-11
    x32 = torch.from_numpy(x).float().cuda()
    assert rel_err(fd.apply(x32).double().cpu().numpy(), ofd.sptime_apply(ref, x)) < 1e-5
