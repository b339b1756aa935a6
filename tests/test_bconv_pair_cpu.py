"""Tensor-core base conversion, host side: the planner's groups and images (bconv_tc_plan.h), their parts, the operand layout and
the kernel's reduction, emulated on the CPU against 128-bit integer arithmetic (tests/bconv_pair_emul.cpp); the rules of its waits (tests/bconv_wait_emul.cpp)."""
import os
import subprocess

import pytest

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(name, tmp_path, *args):
    exe = str(tmp_path / name)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I" + os.path.join(_ROOT, "phantom-fhe_b200", "csrc"),
                           os.path.join(_ROOT, "tests", name + ".cpp"), "-o", exe])
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


@pytest.mark.parametrize("seed", [1, 2026])
def test_pair_image_and_layout_match_big_integer_arithmetic(seed, tmp_path):
    _run("bconv_pair_emul", tmp_path, str(seed))


def test_what_is_in_flight_is_waited_for_after_a_time_out(tmp_path):
    _run("bconv_wait_emul", tmp_path)
