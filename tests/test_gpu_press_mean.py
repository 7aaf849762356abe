"""The pressure's right-hand side of mode (0,0) takes nothing from u and w there: k = 0, and the
mean-flow correction may be writing u(0,0) beside it (tests/press_mean_check.cu)."""
import os
import subprocess

import pytest

from test_fft_host import nvcc

HERE = os.path.dirname(os.path.abspath(__file__))
pytestmark = pytest.mark.gpu


def test_mode_zero_leaves_u_and_w_unread(cuda_ok, tmp_path):
    cc = nvcc()
    if cc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "press_mean_check")
    subprocess.run([cc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(HERE, "press_mean_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    n, bad = (int(x) for x in r.stdout.split())
    assert n > 10000 and bad == 0, (n, bad)
