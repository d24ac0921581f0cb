"""The periodic solve's quotients (divide.cuh) against divisions, on the host
and on the device."""
import ctypes as C
import os
import subprocess

import pytest

from ps3d_b200.build import ARCH, CSRC

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def differ(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("quotients") / "libquotients.so")
    subprocess.run(["nvcc", *ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I" + CSRC,
                    "-shared", "-o", lib, os.path.join(HERE, "quotients.cu")], check=True)
    fn = C.CDLL(lib).quotients_differ
    fn.argtypes = [C.c_int, C.c_int, C.c_ulonglong, C.c_ulonglong]
    fn.restype = C.c_longlong
    return fn


@pytest.mark.parametrize("fp32", [0, 1])
def test_quotients_on_the_host(differ, fp32):
    assert differ(0, fp32, 1 << 21, 5) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("fp32", [0, 1])
def test_quotients_on_the_device(differ, fp32):
    assert differ(1, fp32, 1 << 28, 7) == 0
