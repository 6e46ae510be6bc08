"""Kernels whose launch overlaps their predecessor's end read its output with coherent loads (source check).

The non-coherent path (``__ldg``, ``ld.global.nc``, ``const T* __restrict__``)
promises data that is constant over the grid's life. A kernel launched by
``launch_dependent`` is resident while its predecessor still writes, so the
operands that the predecessor may have written must not go that way: the
vectors of the products and what the Krylov kernels hand on to one another.
"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "qmbed_b200" / "csrc"

# kernel -> operands that the launch before it may have written
OPERANDS = {
    ("tile_rows.cu", "tile_spmv_kernel"): ["x"],
    ("tile_rows.cu", "tile_spmm_kernel"): ["z", "p"],
    ("hv_tile.cu", "exchange_row_kernel"): ["x"],
    ("flipchain.cu", "flip_box_kernel"): ["a.x", "a.p", "a.q"],
    ("flipchain.cu", "flip_group_kernel"): ["a.x", "a.out"],
    ("krylov.cu", "panel_dot_kernel"): ["w"],
    ("krylov.cu", "finish_kernel"): ["partials"],
    ("krylov.cu", "orthogonalize_kernel"): ["h", "beta_device", "src"],
    ("krylov.cu", "scale_and_record_kernel"): ["partials", "h", "src"],
}


def _kernel(file, name):
    source = (CSRC / file).read_text()
    at = re.search(r"__global__[^;{]*?\b" + name + r"\(", source)
    depth, i = 0, source.index("{", at.end())
    for j in range(i, len(source)):
        depth += {"{": 1, "}": -1}.get(source[j], 0)
        if depth == 0:
            return source[at.start():i], source[i:j + 1]
    raise AssertionError(name)


@pytest.mark.parametrize("kernel", sorted(OPERANDS))
def test_operands_of_the_launch_before(kernel):
    signature, body = _kernel(*kernel)
    assert "await_previous();" in body
    for operand in OPERANDS[kernel]:
        assert not re.search(r"__restrict__ " + re.escape(operand) + r"\b", signature), operand
        assert not re.search(r"(__ldg|\bload16)\(\s*(reinterpret_cast<[^>]*>\()?" + re.escape(operand) + r"\b", body), operand


def test_every_dependent_launch_is_listed():
    launched = set()
    for path in CSRC.glob("*.cu"):
        if "await_previous();" not in path.read_text():
            continue
        for match in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(", path.read_text()):
            if "await_previous();" in _kernel(path.name, match.group(1))[1]:
                launched.add((path.name, match.group(1)))
    assert launched == set(OPERANDS)


def test_vector_loads_are_coherent():
    tile_rows, hv_tile = (CSRC / "tile_rows.cu").read_text(), (CSRC / "hv_tile.cu").read_text()
    loader = tile_rows[tile_rows.index("load_complex(const T* x"):]
    assert "__ldg" not in loader[:loader.index("\n}")]
    # the exchange kernel's predicated loads: only the 32-bit table entries are constant
    for element in ("float", "double", "float2", "double2"):
        loader = hv_tile[hv_tile.index(f"load_if(bool on, const {element}* p)"):]
        assert ".nc" not in loader[:loader.index("\n}")], element
