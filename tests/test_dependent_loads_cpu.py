"""Kernels launched with programmatic stream serialisation start while the grid before
them still runs (griddepcontrol.wait orders them). What that grid writes is not
read-only during such a kernel, so it must not be read through the non-coherent path:
no __ldg, no const __restrict__ pointer. A wrong load shows up as a stale line once in
many runs, if at all, so this reads the sources instead."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "igaops_b200" / "csrc"

# file, the load's address as written in the source, how often it is loaded
OPERANDS = [
    ("batch.cu", "partial + (int64_t)b * m + j", 1),  # second stage of the segmented Gram
    ("dense_mode.cuh", "src", 1),  # tensor operand of a dense mode product
    ("fd_tc.cu", "Arow + tailc", 1),  # separate tensor-core products
    ("fd_tc.cu", "Arow + k0 + u", 1),
    ("fd_tc.cu", "reinterpret_cast<const uint4*>(src + (size_t)rr * kp1 + 8 * kc)", 1),
    ("fd_tc.cu", "reinterpret_cast<const uint32_t*>(g.w0 + (size_t)(k0 + j) * R + rr)", 1),
]


@pytest.mark.parametrize("name,address,count", OPERANDS)
def test_operands_of_the_grid_before_are_loaded_coherently(name, address, count):
    text = (CSRC / name).read_text()
    assert text.count("ld_dependent(" + address + ")") == count


def test_no_restrict_qualifier_on_what_the_grid_before_writes():
    batch = (CSRC / "batch.cu").read_text()
    sig = re.search(r"\n    seg_gram_stage2\((.*?)\) \{", batch, re.S).group(1)
    assert re.search(r"const double\* partial\b", sig)
    assert not re.search(r"__restrict__ Arow", (CSRC / "fd_tc.cu").read_text())


def test_every_dependent_launch_is_covered():
    """A new file with a dependent launch comes with its operands in the list above."""
    files = {f.name for f in CSRC.glob("*.cu") if "griddepcontrol.wait" in f.read_text()}
    assert files == {"batch.cu", "dense_mode.cu", "fd_tc.cu", "sptime.cu"}
    # dense_mode.cu and sptime.cu read tensors through stage_elem of dense_mode.cuh
    for name in ("dense_mode.cu", "sptime.cu"):
        text = (CSRC / name).read_text()
        assert not re.search(r"__ldg\(p\.x", text)
        const = re.findall(r"stage_elem<(true|false)>\((?:Xs|dst \+ c \* LDX)", text)
        assert const and set(const) == {"false"}
