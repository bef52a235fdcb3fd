"""The update pass's shared-divisor quotients against divisions, on the host (the
same operations, each rounded as the device rounds it)."""
import os
import shutil
import subprocess

from conftest import ROOT


def test_shared_divisor_is_as_exact_as_a_division(tmp_path):
    exe = str(tmp_path / "divide_check")
    subprocess.run([shutil.which("g++") or "g++", "-O2", "-std=gnu++17", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "spectral_upcxx_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "divide_check.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    worst, tiny = float(out[0]), float(out[1])
    differ, total, special = (int(x) for x in out[2:])
    assert worst <= 0.5 + 2.0 ** -49, worst  # the bound, and the check's own 2^-60
    assert tiny <= 2.0, tiny
    assert differ <= 1e-6 * total, (differ, total)  # only next to a rounding boundary
    assert special == 0
