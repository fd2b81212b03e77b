"""Shared-memory limits belong to a device, and one process may drive several
from as many threads: each device is set up, again after a failure, and not
again after a success."""

import ctypes
import os
import re

import pytest

import native


@pytest.mark.parametrize("devices", [1, 2, 64, 65])
@pytest.mark.parametrize("fails", [0, 2])
def test_every_device_is_set_up(tmp_path, devices, fails):
    lib = native.load("once", tmp_path)
    calls = (ctypes.c_int * devices)()
    lib.once_calls(devices, 1, 5, fails, calls)
    # devices past the flags are set up every time
    assert list(calls) == [fails + 1 if d < 64 else 5 for d in range(devices)]
    lib.once_calls(devices, 4, 5, 0, calls)
    assert all(1 <= c <= (4 if d < 64 else 20) for d, c in enumerate(calls))


def test_no_limit_is_raised_once_per_process():
    for f in ("slq_engine.cu", "slq_mlp.cu"):
        with open(os.path.join(native.CSRC, f)) as s:
            text = s.read()
        assert not re.search(r"static bool \w+ = false;[^}]*"
                             r"cudaFuncSetAttribute", text), f
