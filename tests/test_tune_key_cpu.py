"""Kept tuning entries hit only the kernels and shapes that they were timed on."""
import json
from types import SimpleNamespace

import pytest
import torch

from igaops_b200 import tune


def _plan(**change):
    plan = dict(ndim=3, op=1, st=0, tt=0, tr=0, sym=True, dtype=torch.float64, W=4,
                n=[11, 11, 11], nq=[29, 29, 29], groups=10, P=SimpleNamespace(face=[8, 8]),
                nseg=1)
    plan.update(change)
    plan = SimpleNamespace(**plan)
    plan.set_nseg = lambda k: setattr(plan, "nseg", k)
    return plan


@pytest.fixture
def device(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda: "B200")


def test_face_and_groups_are_part_of_the_shape(device):
    """Rules of the same sizes whose windows move at other points, and other kernels."""
    keys = {tune.shape_key(p) for p in (_plan(), _plan(groups=14),
                                        _plan(P=SimpleNamespace(face=[16, 8])))}
    assert len(keys) == 3


def test_file_of_the_replaced_kernel_is_not_used(device, monkeypatch, tmp_path):
    """Entries without the kernel form (the CTA-per-tile kernel's segment count, and a tile
    kernel that was chosen against it) do not steer the present kernel."""
    old = "|".join(str(v) for v in (3, 1, 0, 0, 0, 1, "float64", 4, 11, 11, 11, 29, 29, 29, "B200"))
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({old: 3, "kernel|" + old: "tile"}))
    monkeypatch.setenv("IGAOPS_B200_TUNE", str(path))
    monkeypatch.setattr(tune, "_LOADED", False)
    monkeypatch.setattr(tune, "_CACHE", {})
    tune._load()
    assert old in tune._CACHE  # the file was read
    key = tune.shape_key(_plan())
    assert key not in tune._CACHE and "kernel|" + key not in tune._CACHE
    # an entry of this form does hit
    tune._CACHE[key] = 5
    plan = _plan()
    assert tune.tune_nseg(plan, None, None, None) == (5, {}) and plan.nseg == 5
