"""The launch knobs' defaults in a new process (no GPU): what programs that put
a knob back by its documented default write."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_defaults():
    from astroviper_b200 import _lib
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("libav200.so not built")
    code = ("from astroviper_b200 import _lib\n"
            "print(*[_lib.lib().av_tune_get(k) for k in range(5)])")
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(v) for v in out] == [16, 16, _lib.AV_GRID_LANES_AUTO, _lib.AV_DEGRID_LANES_AUTO,
                                     _lib.AV_HOGBOM_BARRIER_TIMEOUT_US_DEFAULT]
