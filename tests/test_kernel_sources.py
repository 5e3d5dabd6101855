"""Rules that every kernel source keeps, checked on the text: what they guard against needs more devices, or another
build, than a test has."""

import re

import pytest

from jax_vllm_b200.csrc import build

SOURCES = sorted(build.SRC_DIR.glob("*.cu"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_function_attributes_are_set_on_every_device(path):
    """A function's attributes belong to one device: every cudaFuncSetAttribute stands in the set-up that
    `jv_once_per_device` runs for each device, so that the first launch on a second one finds them."""
    text = path.read_text()
    inside = [m.span() for m in re.finditer(r"jv_once_per_device\(.*?\}\)", text, re.S)]
    for m in re.finditer(r"cudaFuncSetAttribute\(", text):
        line = text.count("\n", 0, m.start()) + 1
        assert any(a < m.start() < b for a, b in inside), f"{path.name}:{line} sets an attribute for one device only"
