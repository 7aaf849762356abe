"""The split Helmholtz solves at the largest channels that run them (below 2432 column segments): 2400
columns, and a multiblock channel of 2256 segments on 1200 columns, where each array of factors and
right-hand sides is used to its end. Bars against the oracle: FP64 1e-12 relative a step (with posts 5e-12 on
the pressure), mixed 1e-5 (1e-4 on the pressure)."""
import numpy as np
import pytest

from oracle import Oracle
from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import initial_field, initial_field_bands, initial_scalars, re_tau_params

pytestmark = pytest.mark.gpu
FIELDS = ("u1", "u2", "u3", "p")


def bar(form, field, posts, step):
    if form == "mixed":
        return 1e-4 if field == "p" else 1e-5
    return (5e-12 if field == "p" and posts else 1e-12) * step


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("posts", [False, True])
def test_2400_columns(cuda_ok, form, posts):
    s = build_setup(re_tau_params(48, 47, Nz=96, posts=posts, post_period=12, post_points=6))
    assert s.ncols == 2400
    st = initial_field(s, 43)
    o, g = Oracle(s), GpuChannel(s, form)
    for x in (o.set_state, g.upload_state):
        x(*st)
    for x in (o, g):
        x.set_scalars(**initial_scalars(s))
    names = g.profile_steps(1)
    assert "k_helm_sweep" in names and "k_helm_uw" not in names
    g.upload_state(*st)
    g.set_scalars(**initial_scalars(s))
    for k in (1, 2):
        o.step()
        g.step()
        g.synchronize()
        for f, x, y in zip(FIELDS, o.get_state(), g.download_state()):
            assert np.linalg.norm(y - x) < bar(form, f, posts, k) * np.linalg.norm(x), (k, f)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_2256_segments_on_1200_columns(cuda_ok, form):
    p = re_tau_params(48, 65)
    p.Ngalx = p.Ngalz = (p.Ngalx[0], 24)
    s = build_setup(p)
    assert s.ncols == 1200 and sum(len(s.band_cols(b)) for b in (1, 2, 3)) == 2256
    f = initial_field_bands(s, 44)
    o, g = Oracle(s), GpuChannel(s, form)
    o.set_bands(f)
    g.upload_bands(f)
    for x in (o, g):
        x.set_scalars(**initial_scalars(s))
    for k in (1, 2):
        o.step()
        g.step()
        g.synchronize()
        ref, got = o.get_bands(), g.download_bands()
        for b in (1, 2, 3):
            for name, x, y in zip(FIELDS, ref[b], got[b]):
                assert np.linalg.norm(y - x) < bar(form, name, False, k) * max(np.linalg.norm(x), 1e-300), (k, b, name)
