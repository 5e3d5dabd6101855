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


@pytest.mark.parametrize("path", SOURCES + sorted(build.SRC_DIR.glob("*.cuh")), ids=lambda p: p.name)
def test_arrays_read_as_vectors_are_aligned_for_them(path):
    """An array of elements that is filled or read sixteen bytes at a time is declared with that alignment (or as vectors):
    in registers it makes no difference, in local memory a vector access off its boundary faults."""
    text = path.read_text()
    arrays = set(re.findall(r"^\s*(?:const )?(?:float|T|TI|TO|TW|W|__nv_bfloat16) (\w+)(?:\[\w+\])+;", text, re.M))
    for kind, name in re.findall(r"reinterpret_cast<(?:const )?(uint4|float4)\*>\(&?(\w+)\b", text):
        assert name not in arrays, f"{path.name}: {name} is read as {kind}, and not aligned for it"
