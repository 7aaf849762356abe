"""The fixed-point transforms of the FP64 form on the CPU (tests/fx_host_check.cu): every
compiled length, both directions, lines of every shape, against a direct DFT in long double
and beside the FP64 Stockham plan."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LENGTHS = (24, 48, 72, 96, 144, 192, 288, 384, 576, 768, 1152)


def test_fixed_point_transforms_against_direct_dft(tmp_path):
    cc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")) if c and os.path.exists(c)), None)
    if cc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fx_host_check")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "cu", os.path.join(HERE, "fx_host_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=900).stdout
    rows = [r.split() for r in out.strip().splitlines()]
    assert {(int(r[0]), int(r[1]), int(r[2])) for r in rows} == {(n, d, s) for n in LENGTHS for d in (0, 1) for s in range(8)}
    for n, d, shape, fixed, fp64, _ in rows:
        # one rounding of each component to FP64 is at most 2^-53 = 1.1e-16 of it; the integer
        # stages may add as much again, and no line may be further off than the FP64 plan
        assert float(fixed) < 2.2e-16, (n, d, shape, fixed)
        assert float(fixed) <= 1.0001 * float(fp64), (n, d, shape, fixed, fp64)
