"""Tensor-core FD apply with the products over directions 1 and 2 in one kernel
(extents up to 128, csrc/fd_tc.cu), against a numpy emulation of its roundings and
against the six separate products."""
import numpy as np
import pytest
import torch

from oracle import fd as ofd
from tests._problems import rules
from tests.test_gpu_fd_geometry import _bf16_apply

pytestmark = pytest.mark.gpu


def _problem(ne):
    """Degree 2, all faces Dirichlet: ne free nodes per direction."""
    from igaops_b200.fastdiag import SingleFD, rewrite_quadrature

    rl = rules(3, 2, ne)
    table = np.ones((1, 3, 2), dtype=bool)
    fd = SingleFD("spatial")
    fd.compute_space_eigendecomposition(rl, table)
    N = int(np.prod([q.nbctrlpts for q in rl]))
    return fd, ofd.setup(rewrite_quadrature(rl), table), N


# extents at the padding's edges (16, 17), at the last small CTA (48, 49), at the
# bound of the path (128) in each direction, ragged ones; 128 x 128 x 3 is also the
# box whose output is cleared by a memset
@pytest.mark.parametrize("ne", [(128, 17, 16), (16, 128, 33), (31, 15, 128), (128, 128, 3),
                                (48, 47, 45), (49, 50, 37), (5, 9, 3)])
@pytest.mark.parametrize("dt,offset", [(torch.float64, 1), (torch.float32, 3)])
def test_fused_tensor_core_apply(cuda, ne, dt, offset):
    """Within 1e-3 (2-norm) of the emulation, which accumulates in FP64: an FP32
    sum off by 1e-6 of its terms rounds to the neighbouring BF16 value (2^-8 off)
    in about one of 10^3 cases, 1.2e-4 rms for each of five roundings.  Entries
    outside the box are zero, whatever the vector held, at any alignment."""
    fd, o, N = _problem(list(ne))
    spfd = fd.space_preconditioner
    assert tuple(spfd._boxes[0][1]) == ne
    x = np.random.default_rng(N).standard_normal(N)
    if dt == torch.float32:
        x = x.astype(np.float32).astype(np.float64)
    buf = torch.full((N + 8,), float("nan"), dtype=dt, device="cuda")
    y = buf[offset:offset + N]
    spfd.apply_device_tc(torch.from_numpy(x).to("cuda", dt), y)
    spfd.check_tc_status()
    got = y.double().cpu().numpy()
    emu = _bf16_apply(o, x)
    assert np.linalg.norm(got - emu) < 1e-3 * np.linalg.norm(emu)
    outside = np.ones(N, dtype=bool)
    outside[spfd.free_nodes(0)] = False
    assert np.all(got[outside] == 0.0)
    assert torch.isnan(buf[:offset]).all() and torch.isnan(buf[offset + N:]).all()


def test_fused_equals_separate_products(cuda):
    """A batch with an extent above 128 runs the separate products for all its
    patches: the same products and roundings, so the same bits.  They use the
    work arrays of a patch's own apply in another layout: values left there that
    are not finite do not reach a later apply, either way."""
    from igaops_b200.fastdiag import MultiFD

    probs = [_problem(ne) for ne in ([6, 7, 9], [128, 17, 16], [31, 49, 20], [130, 4, 5])]
    sizes = [N for _, _, N in probs]
    mfd = MultiFD([fd for fd, _, _ in probs])
    x = torch.from_numpy(np.random.default_rng(5).standard_normal(sum(sizes))).float().cuda()
    y = torch.empty_like(x)
    for _ in range(2):
        for (fd, _, n) in probs:
            bad = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
            fd.space_preconditioner.apply_device_tc(bad, torch.empty_like(bad))
        mfd.apply_device_tc(x, y)
        mfd.apply_device_tc(torch.full_like(x, float("nan")), torch.empty_like(x))
        mfd.check_tc_status()
        start = 0
        for (fd, _, n) in probs:
            one = torch.empty(n, dtype=torch.float32, device="cuda")
            fd.space_preconditioner.apply_device_tc(x[start:start + n].contiguous(), one)
            assert torch.isfinite(one).all()
            assert torch.equal(one, y[start:start + n])
            start += n
