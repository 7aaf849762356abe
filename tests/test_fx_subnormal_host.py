"""The fixed-point transforms of lines of subnormal values on the CPU (tests/fx_subnormal_check.cu): no line
is further off than with the FP64 plan, whose products round to multiples of 2^-1074, and a line of zeros
stays zero."""
import os
import subprocess

import pytest

from test_fft_host import nvcc

HERE = os.path.dirname(os.path.abspath(__file__))
LENGTHS = (24, 48, 72, 96, 144, 192, 288, 384, 576, 768, 1152)


def test_subnormal_lines(tmp_path):
    cc = nvcc()
    if cc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fx_subnormal_check")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "cu", os.path.join(HERE, "fx_subnormal_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=900).stdout
    rows = [r.split() for r in out.strip().splitlines()]
    assert {(int(r[0]), int(r[1]), int(r[2])) for r in rows} == {(n, d, s) for n in LENGTHS for d in (0, 1) for s in range(5)}
    for n, d, shape, fixed, fp64 in rows:
        assert float(fixed) <= float(fp64), (n, d, shape, fixed, fp64)
        assert shape != "4" or float(fixed) == 0
