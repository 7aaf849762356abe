"""The forms of the solves that the autotuner and the batches choose between. All forms of the mixed
Helmholtz solves and of the pressure step give the same bits (tests/solve_variants_check.cu): the
routes are chosen by column counts, and a channel in a batch equals the same channel alone. Tuned
channels that run the fused kernels, alone and in a batch, against the oracle."""
import os
import subprocess

import numpy as np
import pytest

from oracle import Oracle
from rnl_multiblock_nofft_gb300.native import GpuBatch, GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import initial_field, initial_scalars, re_tau_params
from test_fft_host import nvcc

HERE = os.path.dirname(os.path.abspath(__file__))
pytestmark = pytest.mark.gpu
FIELDS = ("u1", "u2", "u3", "p")


def test_every_form_has_the_same_bits(cuda_ok, tmp_path):
    cc = nvcc()
    if cc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "solve_variants_check")
    subprocess.run([cc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(HERE, "solve_variants_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    rows = [[int(x) for x in l.split()] for l in r.stdout.splitlines()]
    assert len(rows) == 6 * 3 * 4 * 3  # shapes, substeps, depths, blocks
    assert all(row[10] == (row[4] == 3) for row in rows)  # the third substep's divergence is there
    bad = [row for row in rows if row[7] or row[8] or row[9]]
    assert not bad, bad


def tuned(s, form, seed):
    st = initial_field(s, seed)
    g = GpuChannel(s, form)
    g.upload_state(*st)
    g.set_scalars(**initial_scalars(s))
    before = g.download_state()
    g.autotune()
    for x, y in zip(before, g.download_state()):
        assert np.array_equal(x, y)
    return g, st


def oracle_steps(s, st, n):
    o = Oracle(s, threads=os.cpu_count() or 1)
    o.set_state(*st)
    o.set_scalars(**initial_scalars(s))
    o.step(n)
    return o.get_state()


def check(ref, got, form, steps):
    for f, x, y in zip(FIELDS, ref, got):
        bar = 1e-12 * steps if form == "fp64" else (1e-4 if f == "p" else 1e-5)
        e = np.linalg.norm(y - x) / np.linalg.norm(x)
        assert e < bar, (f, e)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_tuned_channel_of_18624_columns(cuda_ok, form):
    s = build_setup(re_tau_params(192, 49))
    g, st = tuned(s, form, 51)
    names = g.profile_steps(1).keys()  # (steps once: the fused kernels)
    assert {"k_helm_uw", "k_helm_v", "k_press"} <= set(names) and "k_press_sweep" not in names
    g.upload_state(*st)
    g.set_scalars(**initial_scalars(s))
    g.step(2)
    g.synchronize()
    check(oracle_steps(s, st, 2), g.download_state(), form, 2)
    g.close()


# 2112, 8320 and 8320 columns: fused in the batch, split alone
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_tuned_channels_in_a_batch(cuda_ok, form):
    made = [(s, *tuned(s, form, 60 + i)) for i, s in enumerate(build_setup(re_tau_params(n, ny)) for n, ny in
                                                               ((64, 97), (128, 47), (128, 46)))]
    b = GpuBatch([g for _, g, _ in made])
    b.step(2)
    b.synchronize()
    for s, g, st in made:
        check(oracle_steps(s, st, 2), g.download_state(), form, 2)
    b.close()
