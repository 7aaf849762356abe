"""bench.py's derived figures for the kernels that small channels run and for the FP64 form: every
solve and pressure launch has a byte count, the FP64 form's rate is not read against the FP64
peak, and the triad terms are those that a form sums."""
import os
import sys

import numpy as np
import pytest

import fake_cuda
from rnl_multiblock_nofft_gb300 import build_native
from rnl_multiblock_nofft_gb300.triads import TriadLists, plane_files
from rnl_multiblock_nofft_gb300.workloads import workload_setup

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

SPLIT = ("k_helm_rhs", "k_helm_sweep", "k_press_rhs", "k_press_sweep", "k_press_corr")
PROFILE = """
from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.workloads import workload_setup
g = GpuChannel(workload_setup("C0"), "{form}")
print(" ".join(g.profile_steps(1)))
g.close()
"""


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_small_channels_kernels_have_a_roofline(tmp_path, form):
    build_native.build()
    out, _ = fake_cuda.run(fake_cuda.build(tmp_path), tmp_path / "log", PROFILE.format(form=form))
    names = out.split()
    assert set(SPLIT) <= set(names)
    s = workload_setup("C0")
    for dominant in SPLIT:
        kern = {n: (3, 0.09 if n == dominant else 0.03) for n in names}
        r = bench.kernel_roofline(s, kern, form, None, 6773.0, "measured", "C0")
        assert r["kernel"] == dominant and r["achieved"] > 0 and r["frac"] > 0
    kern = {n: (3, 0.09 if n in SPLIT or n == "k_zfwd_nl" else 0.03) for n in names}
    r = bench.kernel_roofline(s, kern, form, None, 6773.0, "measured", "C0")
    assert set(r["others"]) | {r["kernel"]} == set(SPLIT) | {"k_zfwd_nl"}


def test_split_launches_per_column_level():
    s = workload_setup("C0")
    u, v = bench.column_levels(s, 2), bench.column_levels(s, 1)
    # bytes of a complex value: 16, in the mixed form's nonlinear term 8. Right-hand side: state read, N read and
    # written, the z pass's array read and written, y-flux read, and p once; sweep: right-hand side read, state
    # written (mixed: read too); pressure: psi and the state
    for form, rhs, sweep in (("fp64", 96, 32), ("mixed", 56, 40)):
        assert bench.algorithmic_bytes(s, "k_helm_rhs", form) == (2 * u + v) * rhs + u * 16
        assert bench.algorithmic_bytes(s, "k_helm_sweep", form) == (2 * u + v) * sweep
        assert [bench.algorithmic_bytes(s, k, form) for k in SPLIT[2:]] == [u * 64, u * 56, u * 144]


def test_fp64_rate_has_no_fraction_of_a_peak():
    r = bench.fp64_equivalent_rate(workload_setup("C1"), 38.5)
    assert set(r) == {"flops_per_mode_point", "equivalent_gflops"}


def expanded(a):
    """{target and sources: count} of a list with both z-signs"""
    out = {}
    for la, ka, lp, kp in a.astype(int).tolist():
        for sgn in (1, -1) if ka + kp else (1,):
            k = ((la, sgn * ka), (lp, sgn * kp))
            out[k] = out.get(k, 0) + 1
    return out


def test_triad_terms_of_each_form():
    s = workload_setup("S")
    tl = TriadLists.thinned(s, 0.5, 11)
    fu, fv = plane_files(s)
    all_terms = merged = 0
    for files, types in ((fu[1:-1], ((1, 0), (5, 0), (9, 0), (3, 7))), (fv[1:-1], ((2, 4), (6, 8)))):
        for j in files.tolist():
            for t, t2 in types:
                x = expanded(tl.files[j][t - 1])
                if t2:
                    y = expanded(tl.files[j][t2 - 1])
                    all_terms += sum(x.values()) + sum(y.values())
                    # x's term with the roles exchanged is y's
                    merged += len(set(x) | {(p, a) for a, p in y})
                else:
                    all_terms += sum(x.values())
                    merged += len({frozenset(k) for k in x})
    assert bench.triad_terms(s, tl, "mixed") == all_terms
    assert bench.triad_terms(s, tl, "fp64") == merged
    full = TriadLists.complete(s)
    half = bench.triad_terms(s, full, "fp64") / bench.triad_terms(s, full, "mixed")
    assert 0.5 <= half < 0.51
