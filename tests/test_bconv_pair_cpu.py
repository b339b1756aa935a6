"""Tensor-core base conversion with two coefficients a row: the device image, its parts and the operand layout, emulated on the
CPU against 128-bit integer arithmetic (tests/bconv_pair_emul.cpp)."""
import os
import subprocess

import pytest

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2026])
def test_pair_image_and_layout_match_big_integer_arithmetic(seed, tmp_path):
    exe = str(tmp_path / "bconv_pair_emul")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I" + os.path.join(_ROOT, "phantom-fhe_b200", "csrc"),
                           os.path.join(_ROOT, "tests", "bconv_pair_emul.cpp"), "-o", exe])
    out = subprocess.run([exe, str(seed)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
