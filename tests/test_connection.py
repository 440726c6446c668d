"""The roundings of a geodesic's step are the source's, not the compiler's.

Which of the two geodesic kernels traces a pixel depends on the size of its
launch, and the connection amplifies every rounding by 5e6: the functions of
ipg_connection.cuh, of which both are built, must give the same bits whether a
compiler fuses products and sums or not, and the lanes' shares must add up to
the one-lane form.  Compiled for the host without and with contraction.
"""
import os
import subprocess

import pytest

from ipole_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def bits(tmp_path, name, flags):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-w", "-I", build.CSRC, *flags, os.path.join(HERE, "connection_host.cpp"),
                    "-o", exe, "-lm"], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()


def test_bits_do_not_depend_on_contraction(tmp_path):
    if "fma" not in open("/proc/cpuinfo").read():
        pytest.skip("the host has no fused multiply-add to contract to")
    off = bits(tmp_path, "off", ["-O1", "-ffp-contract=off"])
    fast = bits(tmp_path, "fast", ["-O3", "-mfma", "-ffp-contract=fast"])
    assert off == fast
    assert off[1] == "0", "the lanes' shares differ from the one-lane form"
