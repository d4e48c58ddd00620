"""Kernels that start while their predecessor still runs must not promise that their inputs do not change."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "multimodal_training_b200" / "csrc"
FILES = sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh"))


def _kernels(text):
    """(name, parameters, body) of every kernel"""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\((?:[^()]|\([^()]*\))*\)\s*)*(\w+)\s*\(", text):
        i = m.end()
        depth = 1
        while depth:                       # to the end of the parameters
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, j = text[m.end():i - 1], text.index("{", i)
        k, depth = j + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_inputs_of_overlapped_kernels_are_read_through_ordinary_loads(path):
    for name, params, body in _kernels(path.read_text()):
        if "grid_dependency" not in body:
            continue
        for p in params.split(","):
            assert not ("__restrict__" in p and "const" in p), (name, p)
            if "__restrict__" in p:        # written only
                v = p.split()[-1].lstrip("*")
                assert not re.search(rf"(load8|unpack\w*)\(\s*{v}\b|=\s*\*reinterpret_cast<[^>]*>\({v}\b", body), (name, v)


def test_no_read_only_loads_elsewhere():
    for path in FILES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        assert "__ldg(" not in text and "ld.global.nc" not in text, path.name


def test_every_kernel_is_seen():
    assert sum(len(list(_kernels(p.read_text()))) for p in FILES) >= 30
