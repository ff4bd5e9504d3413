"""Kernel attributes are settled per device (per_device.h), on the CPU: a
process that has run a kernel on device 0 and then runs it on device 1 has to
make the attribute call there too, a failed call is made again, and threads
that meet in it read a settled value. No source may remember such a call in a
plain static flag."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mdsctk_gb300", "csrc")


@pytest.fixture()
def shim(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    out = str(tmp_path / "libperdevice.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I" + CSRC,
                    os.path.join(HERE, "native", "per_device_shim.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


def test_each_device_is_settled_once(shim):
    v = ctypes.c_size_t(0)
    for _ in range(3):
        for device in (0, 1, 7):
            assert shim.per_device_use(device, 0, ctypes.byref(v)) == 0 and v.value == 1000 + device
    assert [shim.per_device_calls(d) for d in (0, 1, 2, 7)] == [1, 1, 0, 1]


def test_a_failed_call_is_made_again(shim):
    v = ctypes.c_size_t(0)
    assert shim.per_device_use(3, -5, ctypes.byref(v)) == -5 and v.value == 0
    assert shim.per_device_use(3, 0, ctypes.byref(v)) == 0 and v.value == 1003
    assert shim.per_device_use(3, -5, ctypes.byref(v)) == 0 and v.value == 1003
    assert shim.per_device_calls(3) == 2


def test_devices_past_the_table(shim):
    v = ctypes.c_size_t(0)
    for _ in range(2):
        assert shim.per_device_use(100, 0, ctypes.byref(v)) == 0 and v.value == 1100
    assert shim.per_device_calls(100) == 2


def test_threads(shim):
    assert shim.per_device_race(8, 4, 20000) == 0


def test_no_process_wide_attribute_flags():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            src = open(os.path.join(CSRC, f)).read()
            assert not re.search(r"static\s+bool\s+\w+\s*(=\s*false)?;", src), f
