"""The mixed form's log / atan (log_fast, atan_fast of sc_ddmath.cuh: the
quick evaluations rounded once, without a rounding test), and both forms' on
the device."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "src_b200", "csrc")


def _tool(*paths):
    return next((p for p in paths if p and os.path.exists(p)), None)


def test_fast_log_and_atan_errors(tmp_path):
    """Half an ulp for the rounding, and of the evaluation's error (2^-66.3
    for log, 2^-67.5 of the value for atan): below 2^-15 ulp for |log x| >= 2
    and for atan, 2^-6.3 ulp where |log x| is as small as 2^-8 (nearer 1 the
    table entry is 1 and the error falls with the value)."""
    cxx = _tool("/usr/bin/g++", shutil.which("g++"))
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "fast")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, os.path.join(HERE, "ddmath_fast_check.cpp"),
                    "-o", exe, "-lquadmath"], check=True)
    far, everywhere, at = map(float, subprocess.run([exe, "500000"], check=True, capture_output=True, text=True).stdout.split())
    assert 0.49 < far <= 0.5001 and 0.49 < at <= 0.5001
    assert everywhere <= 0.513


@pytest.mark.gpu
def test_device_log_and_atan(gpu, tmp_path):
    """log_dd, atan_dd: the full evaluation's bits and the host's.  log_fast
    has no device branch: the host's bits.  atan_fast (its own reciprocal):
    never further than the neighbour, and off only where the value lies within
    its error (2^-14 ulp on each side of a tie, so below 2^-12 of the
    arguments).  The reciprocal: 2^-20 cubed, plus the roundings."""
    nvcc = _tool("/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
    assert nvcc, "the check is built with nvcc"
    exe = str(tmp_path / "device")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-O2,-ffp-contract=off", "-diag-suppress", "20091", "-I", CSRC, os.path.join(HERE, "ddmath_device_check.cu"),
                    os.path.join(HERE, "ddmath_host_eval.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000"], check=True, capture_output=True, text=True).stdout.split()
    n, log_full, atan_full, log_host, atan_host, fast_host, far, off = map(int, out[:8])
    assert n == 2_000_000
    assert (log_full, atan_full, log_host, atan_host, fast_host) == (0, 0, 0, 0, 0), out
    assert far == 0 and off < n / 4096, out
    assert float(out[8]) < 2.0 ** -51, out
