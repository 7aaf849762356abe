"""A multiblock channel whose core band is much coarser than its thin wall bands: nearly two column
segments per column, so the split pressure step's faces are more than the transforms' scratch holds.

Bars: against the oracle after one step those of the multiblock tests (FP64 1e-12 relative, the
pressure with posts 5e-12; mixed 1e-5 and, for the pressure, 1e-4); the channel alone (split
pressure step) equals the same channel in a batch that runs the fused one, bit for bit, the
largest divergence included."""
import os

import numpy as np
import pytest

from oracle import Oracle
from rnl_multiblock_nofft_gb300.native import GpuBatch, GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import initial_field_bands, initial_scalars, re_tau_params

pytestmark = pytest.mark.gpu
FIELDS = ("u1", "u2", "u3", "p")


def thin_bands():
    p = re_tau_params(96, 129, Nz=128, posts=True, post_period=24, post_points=12, post_height_plus=0.3)
    p.Ngalx, p.Ngalz = (p.Ngalx[0], 24), (p.Ngalz[0], 48)
    return build_setup(p)


def channel(s, form, f):
    g = GpuChannel(s, form)
    g.upload_bands(f)
    g.set_scalars(**initial_scalars(s))
    return g


@pytest.mark.parametrize("form,vel,press", [("fp64", 1e-12, 5e-12), ("mixed", 1e-5, 1e-4)])
def test_thin_wall_bands(cuda_ok, form, vel, press):
    s = thin_bands()
    f = [initial_field_bands(s, 61 + i) for i in range(2)]
    o = Oracle(s, threads=os.cpu_count() or 1)
    o.set_bands(f[0])
    o.set_scalars(**initial_scalars(s))
    o.step()
    alone, batched = [channel(s, form, x) for x in f], [channel(s, form, x) for x in f]
    b = GpuBatch(batched)
    b.step()
    b.synchronize()
    for g in alone:
        g.step()
        g.synchronize()
    ref, got = o.get_bands(), alone[0].download_bands()
    for band in (1, 2, 3):
        for name, x, y in zip(FIELDS, ref[band], got[band]):
            e = np.linalg.norm(y - x) / max(np.linalg.norm(x), 1e-300)
            assert e < (press if name == "p" else vel), (band, name, e)
    for ga, gb in zip(alone, batched):
        x, y = ga.download_bands(), gb.download_bands()
        for band in (1, 2, 3):
            for name, u, v in zip(FIELDS, x[band], y[band]):
                assert np.array_equal(u, v), (band, name)
        assert ga.scalars() == gb.scalars()
