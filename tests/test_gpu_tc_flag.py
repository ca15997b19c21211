"""The timeout flag of the tensor-core kernels is cleared in the order of the stream that read it: a call on a
stream of its own after one that timed out must not see the old flag, however busy the default stream is."""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_flag_is_cleared_before_the_next_read(agb, tmp_path):
    import os
    from aurora_gb300 import build
    here = os.path.dirname(os.path.abspath(__file__))
    lib = str(tmp_path / "libtc_flag_probe.so")
    subprocess.check_call([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-shared", "-o", lib,
                           os.path.join(here, "cpp", "tc_flag_probe.cu"), "-lcudart"])
    flags = (ctypes.c_int * 2)(-1, -1)
    assert ctypes.CDLL(lib).tc_flag_probe(flags) == 0
    assert list(flags) == [1, 0]
