"""The solves' and the pressure step's routes at the sizes where they change. Channels of few
columns run both as split launches; larger ones, and batches with many columns in flight, run
the fused kernels.

Bars: a channel in a batch equals the same channel alone bit for bit in the mixed form, whichever
route the pressure step takes (it does the same operations in the same order); in the FP64 form
too, for the Helmholtz route follows the channel's own size. Against the oracle the FP64 form is
within 1e-12 relative a step."""
import numpy as np
import pytest

from oracle import Oracle
from rnl_multiblock_nofft_gb300.native import GpuBatch, GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import initial_field, initial_scalars, re_tau_params

pytestmark = pytest.mark.gpu
FIELDS = ("u1", "u2", "u3", "p")


def channel(s, form, st):
    g = GpuChannel(s, form)
    g.upload_state(*st)
    g.set_scalars(**initial_scalars(s))
    return g


# 8320 and 4704 columns: alone below 16384 (split pressure), together above it; 2112, 1200 and 544:
# alone below 2432 (split solves of the mixed form), together above it
@pytest.mark.parametrize("form,sizes,flpress,ny,posts", [
    ("mixed", (128, 128, 96), 0, 45, False), ("mixed", (128, 128, 96), 1, 46, False),
    ("fp64", (128, 128, 96), 0, 46, False), ("fp64", (128, 128, 96), 1, 45, False),
    ("mixed", (64, 48, 32), 0, 46, True), ("mixed", (64, 48, 32), 1, 45, False)])
def test_split_and_fused_routes_agree(cuda_ok, form, sizes, flpress, ny, posts):
    alone, batched = [], []
    for i, n in enumerate(sizes):
        s = build_setup(re_tau_params(n, ny + i, flpress=flpress, posts=posts, post_period=12, post_points=6))
        st = initial_field(s, 700 + i)
        alone.append(channel(s, form, st))
        batched.append(channel(s, form, st))
    b = GpuBatch(batched)
    b.step(2)
    b.synchronize()
    for ga, gb in zip(alone, batched):
        ga.step(2)
        ga.synchronize()
        for f, x, y in zip(FIELDS, ga.download_state(), gb.download_state()):
            assert np.array_equal(x, y), f
        assert ga.scalars() == gb.scalars()


# 2112, 2401 (the largest below 2432) and 3168 columns, levels not a multiple of the kernels' 8
@pytest.mark.parametrize("nx,nz,ny,posts", [(64, 64, 45, False), (96, 48, 47, True), (64, 96, 45, True)])
def test_helmholtz_routes_match_oracle(cuda_ok, nx, nz, ny, posts):
    s = build_setup(re_tau_params(nx, ny, Nz=nz, posts=posts, post_period=12, post_points=6))
    st = initial_field(s, 41)
    o = Oracle(s)
    o.set_state(*st)
    o.set_scalars(**initial_scalars(s))
    g = channel(s, "fp64", st)
    for k in range(2):
        o.step()
        g.step()
        g.synchronize()
        for f, x, y in zip(FIELDS, o.get_state(), g.download_state()):
            assert np.linalg.norm(y - x) < 1e-12 * (k + 1) * np.linalg.norm(x), (k, f)
