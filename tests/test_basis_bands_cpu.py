"""Bands of a rule's basis matrices follow the matrices, not the rule object: a rule whose
basis is replaced (either matrix) gets the bands of the new one."""
import numpy as np
import pytest
import scipy.sparse as sp

from igaops_b200.bands import basis_band
from tests._problems import rules


def _dense(band, cols):
    start, vals = band[0], band[1]
    out = np.zeros((2, len(start), cols + vals[0].shape[1]))
    for r, s in enumerate(start):
        for k in range(2):
            out[k, r, s:s + vals[k].shape[1]] = vals[k][r]
    return out[:, :, :cols]


@pytest.mark.parametrize("which", [(0,), (1,), (0, 1)])
def test_replaced_basis_gets_new_bands(which):
    q = rules(1, 3, 5)[0]
    old = [b.toarray() for b in q.basis]
    assert np.array_equal(_dense(basis_band(q), q.nbctrlpts), old)
    assert basis_band(q) is basis_band(q)
    for k in which:
        q.basis[k] = sp.csr_array((k + 2.0) * q.basis[k])
    new = [b.toarray() for b in q.basis]
    assert np.array_equal(_dense(basis_band(q), q.nbctrlpts), new)
