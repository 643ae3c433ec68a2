"""Dense mode products and the FD apply on them at the edges of their tiles:
extents around the 8-row blocks and the k-steps of four, the limits of the
two-stage launch and of the shared-memory staging, every tensor dimension,
several columns, both orientations of the factor, accumulation; against numpy in
FP64.  Tolerances (relative max norm): FP64 1e-12 -- sums of at most 400 products
of O(1) terms round below 400 x 1.1e-16 x the largest partial sum -- and FP32
1e-5, the tolerance of the other FP32 operators (inputs and results rounded to
2^-24, sums in FP64)."""
import ctypes

import numpy as np
import pytest
import torch

from tests._problems import rel_err

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-12, torch.float32: 1e-5}


def _orthogonal(rng, m):
    return np.linalg.qr(rng.standard_normal((m, m)))[0]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("outer,rows,cols,inner", [
    (1, 1, 1, 1), (3, 5, 4, 1), (1, 8, 9, 65), (2, 33, 7, 64), (70, 17, 31, 3),
    (9, 64, 65, 1), (1, 300, 384, 17), (2, 12, 385, 5), (1, 129, 97, 200)])
def test_mode_product(cuda, outer, rows, cols, inner, dtype):
    from igaops_b200 import MatrixFree

    rng = np.random.default_rng(rows * 1000 + cols)
    A = rng.standard_normal((rows, cols))
    x = rng.standard_normal((outer, cols, inner))
    xt = torch.from_numpy(x).cuda().to(dtype)
    got = MatrixFree.tensor_matrix_product(xt, A, 1).cpu().numpy()
    assert rel_err(got, np.einsum("rc,oci->ori", A, x)) < TOL[dtype]
    y = rng.standard_normal((outer, rows, inner))
    yt = torch.from_numpy(y).cuda().to(dtype)
    back = MatrixFree.tensor_matrix_product(yt, A, 1, is_transpose=True).cpu().numpy()
    assert rel_err(back, np.einsum("rc,ori->oci", A, y)) < TOL[dtype]


def test_mode_product_accumulates(cuda):
    from igaops_b200 import _lib
    from igaops_b200._device import stream_handle
    from igaops_b200.bands import DeviceFactor

    rng = np.random.default_rng(5)
    A, x, y = rng.standard_normal((11, 13)), rng.standard_normal((2, 13, 70)), \
        rng.standard_normal((2, 11, 70))
    f = DeviceFactor(A, torch.float64, False)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    _lib.check(_lib.LIB.iga_mode_product(_lib.IGA_F64, f.f, 2, 70, xd.data_ptr(), yd.data_ptr(), 1,
                                         stream_handle()))
    assert rel_err(yd.cpu().numpy(), y + np.einsum("rc,oci->ori", A, x)) < 1e-12


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,ncols", [
    ([1], 1), ([7], 2), ([130], 1), ([5, 9], 1), ([64, 136], 1), ([3, 137], 1), ([150, 160], 1),
    ([8, 7, 9], 1), ([1, 33, 2], 1), ([17, 16, 15], 3), ([12, 4, 129], 1), ([40, 3, 137], 1),
    ([4, 3, 2, 5], 1), ([3, 2, 4, 2], 2), ([6, 2, 390], 1)])
def test_fd_apply_edges(cuda, m, ncols, dtype):
    """iga_fd_apply on a box inside a larger tensor: the box is gathered, entries
    outside it (NaN) are never read, and the result is zero outside it."""
    from igaops_b200 import _lib
    from igaops_b200._device import iga_dtype, stream_handle

    rng = np.random.default_rng(sum(m) + ncols)
    nd = len(m)
    lo = [int(k % 2) for k in range(nd)]
    n = [mm + l + 1 for mm, l in zip(m, lo)]
    U = [_orthogonal(rng, mm) for mm in m]
    lam = rng.uniform(0.5, 2.0, m[::-1])
    box = tuple(slice(l, l + mm) for l, mm in zip(lo, m))[::-1]
    x = np.full(n[::-1] + [ncols], np.nan)
    x[box] = rng.standard_normal(m[::-1] + [ncols])
    t = x[box]
    for d in range(nd):
        t = np.moveaxis(np.tensordot(U[d].T, t, axes=(1, nd - 1 - d)), 0, nd - 1 - d)
    t = t / lam[..., None]
    for d in range(nd):
        t = np.moveaxis(np.tensordot(U[d], t, axes=(1, nd - 1 - d)), 0, nd - 1 - d)
    ref = np.zeros_like(x)
    ref[box] = t
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(dtype)
    xd, Ud, inv = dev(x), [dev(u) for u in U], dev(1.0 / lam)
    yd = torch.full_like(xd, 7.0)
    w = [torch.empty(t.size, dtype=dtype, device="cuda") for _ in range(2)]
    arr = ctypes.c_int32 * nd
    ptr = (ctypes.c_void_p * nd)(*[u.data_ptr() for u in Ud])
    _lib.check(_lib.LIB.iga_fd_apply(iga_dtype(dtype), nd, arr(*n), arr(*lo), arr(*m), ptr,
                                     inv.data_ptr(), ncols, xd.data_ptr(), yd.data_ptr(),
                                     w[0].data_ptr(), w[1].data_ptr(), stream_handle()))
    assert rel_err(yd.cpu().numpy(), ref) < TOL[dtype]
