"""The split pressure step's array of the faces below its chunks, on the CPU: every launch that uses
it gets room for one complex value per column segment and chunk of levels, whatever the bands.

Channels with a core much coarser than thin wall bands have nearly two column segments per column,
so this array can be the larger one beside the transforms' scratch (192 x 64, core 16 x 16, ny 385,
posts of 0.3 wall units: 9.6 MB beside 6.7 MB)."""
import pytest

import fake_cuda
from rnl_multiblock_nofft_gb300 import build_native

CODE = """
from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import re_tau_params
p = re_tau_params({nx}, {ny}, Nz={nz}, posts={posts} > 0, post_period=24, post_points=12, post_height_plus={posts} or 6.0)
p.Ngalx, p.Ngalz = (p.Ngalx[0], 3 * {cx} // 2), (p.Ngalz[0], 3 * {cz} // 2)
s = build_setup(p)
g = GpuChannel(s, "{form}")
for k in (1, 2, 3):
    g.substep(k)
print(sum(len(s.band_cols(b)) for b in (1, 2, 3)))
g.close()
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build_native.build()
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


# wall band, core band, levels, post height (wall units; 0: no posts): thin wall bands under coarse
# cores first, then cores half as wide and as wide as the wall bands'
@pytest.mark.parametrize("form", ["mixed", "fp64"])
@pytest.mark.parametrize("nx,nz,cx,cz,ny,posts", [
    (192, 64, 16, 16, 385, 0.2), (192, 64, 16, 16, 385, 0.3), (192, 64, 16, 16, 385, 0.4), (128, 96, 16, 16, 385, 0.3),
    (96, 128, 16, 32, 129, 0.3), (96, 96, 16, 16, 201, 0.5), (96, 96, 32, 16, 97, 0), (64, 64, 32, 32, 129, 6.0),
    (32, 32, 16, 16, 65, 0), (64, 64, 64, 64, 65, 0), (16, 16, 16, 16, 41, 0)])
def test_faces_fit_their_array(fake, tmp_path, form, nx, nz, cx, cz, ny, posts):
    out, log = fake_cuda.run(fake, tmp_path / "log", CODE.format(nx=nx, nz=nz, cx=cx, cz=cz, ny=ny, posts=posts, form=form),
                             "k_press_rhs:5,k_press_corr:6")
    nvc = int(out)
    assert nvc < 16384
    rhs, corr = fake_cuda.launches(log, "k_press_rhs"), fake_cuda.launches(log, "k_press_corr")
    assert len(rhs) == len(corr) == 3
    assert [a[4] != 0 for _, _, a in rhs] == [False, False, True]  # the third substep alone uses it
    for _, grid, args in (rhs[2], corr[2]):
        faces = args[4] if args is rhs[2][2] else args[5]
        assert faces == rhs[2][2][4]
        # index chunk * nvc + segment, chunk < grid y: 16 bytes each
        need = 16 * grid[1] * nvc
        room = [a + n - faces for a, n in fake_cuda.allocations(log) if a <= faces < a + n]
        assert len(room) == 1 and need <= room[0], (need, room)
