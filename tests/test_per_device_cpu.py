"""What the library remembers of a device (shared-memory opt-ins, the number of
multiprocessors) is kept per device and is safe between threads.  (The library
itself has not run on a second GPU.)"""
import ctypes
import glob
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "arbor-cuda_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("per_device") / "per_device.so")
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-I", CSRC, os.path.join(HERE, "emu", "per_device.cpp"),
                    "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("devices", [1, 2, 8, 64])
def test_found_once_per_device(lib, devices):
    assert lib.finds(devices, 5) == devices


def test_devices_past_the_table_are_asked_every_time(lib):
    assert lib.finds(66, 3) == 64 + 2 * 3


def test_a_failure_is_not_kept(lib):
    assert lib.finds_after_failures(2, 6) == 3


def test_threads(lib):
    assert lib.wrong_answers(8, 16) == 0


def test_no_flag_without_a_device():
    """No function keeps a device's state in a static that has no device."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.h")):
        with open(path) as f:
            found = re.findall(r"^\s+static (?:bool|int|const void\*) \w+.*", f.read(), re.M)
        assert not found, f"{os.path.basename(path)}: {found}"
