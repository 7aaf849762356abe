"""What may run beside the mean-flow correction, on the CPU: it changes u(0,0) at every level, so only
kernels that leave u(0,0) alone may: the mixed form's solves of the other modes (mode (0,0) has its
own, before), the reset of the divergence maximum, and the pressure's right-hand side and sweep."""
import pytest

import fake_cuda
from rnl_multiblock_nofft_gb300 import build_native

CODE = """
from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import re_tau_params
s = build_setup(re_tau_params({nx}, {ny}, Nz={nz}, flpress={flpress}, posts={posts}, post_period=8, post_points=4,
                              post_height_plus=20.0))
g = GpuChannel(s, "{form}")
for k in (1, 2, 3, 1, 2, 3):
    g.substep(k)
g.close()
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build_native.build()
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


BESIDE = ("k_helm_rhs_mx", "k_helm_sweep_mx", "k_helm_u_mx", "k_reset_err", "k_press_rhs", "k_press_sweep")


# 144, 544 and 3136 columns: split solves and pressure, fused solves and split pressure; 18624: fused
@pytest.mark.parametrize("form", ["mixed", "fp64"])
@pytest.mark.parametrize("nx,nz,ny,flpress,posts", [(16, 16, 41, 0, False), (32, 32, 65, 0, True), (96, 64, 47, 0, False),
                                                   (192, 192, 33, 0, False), (32, 32, 65, 1, False)])
def test_beside_the_mean_flow(fake, tmp_path, form, nx, nz, ny, flpress, posts):
    _, log = fake_cuda.run(fake, tmp_path / "log", CODE.format(nx=nx, nz=nz, ny=ny, flpress=flpress, posts=posts, form=form))
    runs, beside = fake_cuda.concurrent(log, "k_meanflow")
    assert len(runs) == (0 if flpress else 6)
    assert all(any(b in k for b in BESIDE) for k in beside), beside
