"""The handle's plane transforms over the number range, with bars that do not grow with the plane, and
on planes of subnormal values.

Bars. Against NumPy's transform: relative L2 error 4e-15 and largest error over the plane's largest
value 1e-14. (The fixed-point passes are within 2.2e-16 of a line's L2 norm in each direction, NumPy's
within about 0.6 log2(N) 2^-53 = 7e-16 at 1152: 1.8e-15 for the two directions of both, and the largest
error of a plane is a few times its rms.) Subnormal planes, against
NumPy's transform of the planes times 2^1074 (exact), in units d = 2^-1074: a pass is within 16 d
(tests/fx_subnormal_check.cu: at most 11.9 at any length). Inverse: a line of the second pass sums less than
G1 complex values of the first: 16 sqrt(2) G1 d, and 16 d of its own. Forward: such sums are divided by
G1 G2, which leaves the rounding of the result: 2 d."""
import numpy as np
import pytest

from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import re_tau_params
from test_gpu_fx_leaves import to_modes, to_points

pytestmark = pytest.mark.gpu


def transforms(nx, nz, spec, phys):
    import torch
    g = GpuChannel(build_setup(re_tau_params(nx, 49, Nz=nz)), "fp64")
    d_spec, d_phys = torch.from_numpy(spec).cuda(), torch.from_numpy(phys).cuda()
    o_phys, o_spec = torch.full_like(d_phys, 7.0), torch.full_like(d_spec, 7.0)
    torch.cuda.synchronize()
    g.four_to_phys(d_spec.data_ptr(), o_phys.data_ptr(), len(spec))
    g.phys_to_four(d_phys.data_ptr(), o_spec.data_ptr(), len(phys))
    g.synchronize()
    out = o_phys.cpu().numpy(), o_spec.cpu().numpy()
    g.close()
    return out


# x and z lengths 24 ... 1152, every plan among them
@pytest.mark.parametrize("nx,nz", [(16, 768), (32, 192), (48, 96), (64, 512), (96, 16), (128, 384), (192, 32), (256, 48),
                                   (384, 128), (512, 64), (768, 256)])
def test_error_does_not_grow_with_the_plane(cuda_ok, nx, nz):
    gx, gz = 3 * nx // 2, 3 * nz // 2
    rng = np.random.default_rng(nx * 1000 + nz + 1)
    scales = np.array([1.0, 1e-290, 1e290, 3e-300, 1.0, 1.0])
    n = len(scales)
    spec = rng.normal(size=(n, nz, nx // 2 + 1)) + 1j * rng.normal(size=(n, nz, nx // 2 + 1))
    spec[4] *= np.exp(-np.arange(nx // 2 + 1) * 40.0 / nx)[None, :]   # decaying, one mode of order one
    spec[4, 0, 0] = 1.5
    spec[5] = 0
    spec[5, 1, 2] = 0.25 + 0.5j                                        # a single mode
    phys = rng.normal(size=(n, gz, gx))
    phys[4] = 1.0 + 1e-6 * phys[4]                                     # nearly constant
    phys[5] *= 1e-9
    phys[5, 3, 4] = 2.0                                                # a spike
    got_p, got_s = transforms(nx, nz, spec * scales[:, None, None], phys * scales[:, None, None])
    for got, ref in ((got_p, to_points(spec, gx, gz)), (got_s, to_modes(phys, nx, nz))):
        for i in range(n):
            e = got[i] / scales[i] - ref[i]
            assert np.linalg.norm(e) < 4e-15 * np.linalg.norm(ref[i]), (i, np.linalg.norm(e) / np.linalg.norm(ref[i]))
            assert np.abs(e).max() < 1e-14 * np.abs(ref[i]).max(), (i, np.abs(e).max() / np.abs(ref[i]).max())


@pytest.mark.parametrize("nx,nz", [(16, 768), (96, 16), (64, 96), (256, 48), (768, 32)])
def test_subnormal_planes(cuda_ok, nx, nz):
    gx, gz, d = 3 * nx // 2, 3 * nz // 2, 2.0 ** -1074
    rng = np.random.default_rng(nx + nz)
    scales = np.array([1e-311, 1e-318, 0.0])
    spec = (rng.normal(size=(3, nz, nx // 2 + 1)) + 1j * rng.normal(size=(3, nz, nx // 2 + 1))) * scales[:, None, None]
    phys = rng.normal(size=(3, gz, gx)) * scales[:, None, None]
    assert np.abs(spec).max() < 2.0 ** -1022 and np.abs(phys).max() < 2.0 ** -1022
    got_p, got_s = transforms(nx, nz, spec, phys)
    # in multiples of d
    unit = lambda x: (x * 2.0 ** 537) * 2.0 ** 537
    ep = unit(got_p) - to_points(unit(spec), gx, gz)
    es = unit(got_s) - to_modes(unit(phys), nx, nz)
    assert np.abs(ep).max() < 16 * (1.5 * gx + 1) + 1e-14 * np.abs(to_points(unit(spec), gx, gz)).max(), np.abs(ep).max()
    assert max(np.abs(es.real).max(), np.abs(es.imag).max()) < 2 + 1e-14 * np.abs(to_modes(unit(phys), nx, nz)).max()
    assert not got_p[2].any() and not got_s[2].any()
