"""Alignment and size of device data, checked by compiling device_layout.cu against the library's header."""
import os
import subprocess

import build as pkg_build  # gpu-svdag-editing_b200/build.py

HERE = os.path.dirname(os.path.abspath(__file__))


def test_zero_item_is_aligned_for_wide_loads(tmp_path):
    """item_ptr answers a bad handle with a zero item instead of faulting; phases that read items in 16-byte
    words would fault on one that is aligned for 4-byte words only."""
    cmd = [pkg_build.NVCC, *pkg_build.NVCC_FLAGS, "-I", pkg_build.CSRC, "-c", os.path.join(HERE, "device_layout.cu"), "-o",
           str(tmp_path / "device_layout.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
