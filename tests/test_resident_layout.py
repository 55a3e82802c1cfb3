"""Layout rules of the resident integrator's buffers, over all shapes, on the host.

tests/cuda/resident_layout.cu compiles the rules that the kernel itself uses (kura_resident.cuh)."""
import os
import subprocess

import pytest

from kuramoto_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def layout_bin(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("layout") / "resident_layout")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.INC, "-I", build.SRC,
                    os.path.join(HERE, "cuda", "resident_layout.cu"), "-o", out], check=True, capture_output=True,
                   timeout=600)
    return out


@pytest.mark.parametrize("rule", ["part", "slices"])
def test_rule_holds_for_every_shape(layout_bin, rule):
    r = subprocess.run([layout_bin, rule], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
