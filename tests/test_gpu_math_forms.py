"""The device's shorter arithmetic forms, on every argument they can be given.

csrc/math_check.cu compares them on the GPU with the IEEE operation or the shared
math layer's function that they stand for (exhaustively, so no tolerance).
"""

import subprocess

import pytest

from tractography_b200._lib import LIB_PATH

pytestmark = pytest.mark.gpu

ARGUMENTS = {"tgm_rcp": 250 << 23, "rcp_signed": 1 << 32, "sqrt_pos2_draws": (1 << 24) - 1,
             "sqrt_pos": 1 << 24, "sqrt_pos2_mantissas": 2 << 23, "log_pos2": (1 << 24) - 1, "cos2pi_2": 1 << 32,
             "exps2": 0x3f800001, "softmax": 1 << 32}


def test_forms_equal_what_they_stand_for(runtime):
    out = subprocess.run([LIB_PATH.parent / "math_check"], capture_output=True, text=True, timeout=120, check=True)
    lines = {name: (int(tried), int(bad)) for name, tried, bad in (line.split() for line in out.stdout.splitlines())}
    assert lines == {name: (tried, 0) for name, tried in ARGUMENTS.items()}
