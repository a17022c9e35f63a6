"""Kernels launched while the launch before them ends (early_launch.cuh): what they read was
written by that launch, so no pointer of theirs may promise the compiler constant memory."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "realcausticsengine_gb300" / "csrc"


def _early_kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for name in sorted(set(re.findall(r"launch_early\(\s*(\w+)", text))):
            yield path.name, name, text


@pytest.mark.parametrize("file,name,text", [pytest.param(*k, id=f"{k[0]}:{k[1]}") for k in _early_kernels()])
def test_early_launched_kernels_read_plain_memory(file, name, text):
    m = re.search(r"__global__[^;{]*?\b" + name + r"\s*\(([^{;]*)\)\s*\{", text)
    assert m, f"{name}: definition not found in {file}"
    assert "__restrict__" not in m.group(1)
    body = text[m.end():text.index("\n}\n", m.end())]
    assert "early_launch_wait();" in body
    assert "__ldg(" not in body and "ld.global.nc" not in body


def test_early_launched_kernels_are_found():
    assert {n for _, n, _ in _early_kernels()} >= {"k_mlp_train", "k_reduce_adam", "k_hist", "k_partition", "k_smem_build"}
