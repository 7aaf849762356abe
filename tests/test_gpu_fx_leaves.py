"""The handle's plane transforms (fixed point inside) at the edges of the number range and on
lines with Inf or NaN, against the same transform in NumPy."""
import numpy as np
import pytest

from rnl_multiblock_nofft_gb300.native import GpuChannel
from rnl_multiblock_nofft_gb300.setup_grid import build_setup
from rnl_multiblock_nofft_gb300.workloads import re_tau_params

pytestmark = pytest.mark.gpu


def to_points(x, gx, gz):
    n2 = x.shape[-2]
    a = np.zeros((*x.shape[:-2], gz, x.shape[-1]), complex)
    a[..., :n2 // 2, :] = x[..., :n2 // 2, :]
    a[..., gz - n2 // 2:, :] = x[..., n2 // 2:, :]
    return np.fft.irfft(np.fft.ifft(a, axis=-2, norm="forward"), n=gx, axis=-1, norm="forward")


def to_modes(f, n1, n2):
    x = np.fft.fft(np.fft.rfft(f, axis=-1, norm="forward")[..., :n1 // 2 + 1], axis=-2, norm="forward")
    return np.concatenate([x[..., :n2 // 2, :], x[..., f.shape[-2] - n2 // 2:, :]], axis=-2)


# x and z lengths 24 ... 1152, every plan among them
@pytest.mark.parametrize("nx,nz", [(16, 768), (32, 192), (48, 96), (64, 512), (96, 16), (128, 384), (192, 32), (256, 48),
                                   (384, 128), (512, 64), (768, 256)])
def test_leaves_over_the_number_range(cuda_ok, nx, nz):
    import torch
    g = GpuChannel(build_setup(re_tau_params(nx, 49, Nz=nz)), "fp64")
    gx, gz = 3 * nx // 2, 3 * nz // 2
    rng = np.random.default_rng(nx * 1000 + nz)
    scales = [1.0, 1e-290, 1e290, 3e-300, 0.0, 1.0, 1.0]
    n = len(scales)
    spec = (rng.normal(size=(n, nz, nx // 2 + 1)) + 1j * rng.normal(size=(n, nz, nx // 2 + 1)))
    for i, s in enumerate(scales):
        spec[i] *= s
    spec[5] *= np.exp(-np.arange(nx // 2 + 1) * 40.0 / nx)[None, :]   # decaying, one mode of order one
    spec[5, 0, 0] = 1.5
    spec[6] = 0
    spec[6, 1, 2] = 0.25 + 0.5j                                        # a single mode
    phys = rng.normal(size=(n, gz, gx)) * np.array(scales)[:, None, None]
    phys[5] = 1.0 + 1e-6 * phys[5]                                     # nearly constant
    phys[6] *= 1e-9
    phys[6, 3, 4] = 2.0                                                # a spike
    d_spec, d_phys = torch.from_numpy(spec).cuda(), torch.from_numpy(phys).cuda()
    o_phys, o_spec = torch.full_like(d_phys, 7.0), torch.full_like(d_spec, 7.0)
    torch.cuda.synchronize()
    g.four_to_phys(d_spec.data_ptr(), o_phys.data_ptr(), n)
    g.phys_to_four(d_phys.data_ptr(), o_spec.data_ptr(), n)
    g.synchronize()
    for got, ref in ((o_phys.cpu().numpy(), to_points(spec, gx, gz)), (o_spec.cpu().numpy(), to_modes(phys, nx, nz))):
        for i in range(n):
            # both sides round in FP64: 1e-14 of the plane's norm, the bar of the leaf parity tests
            # being 1e-13
            norm = max(np.abs(ref[i]).max(), 1e-300)
            assert np.abs(got[i] / norm - ref[i] / norm).max() < 1e-14 * np.sqrt(ref[i].size), (i, scales[i])
    g.close()


def test_leaves_carry_nonfinite_lines(cuda_ok):
    import torch
    nx, nz = 64, 96
    g = GpuChannel(build_setup(re_tau_params(nx, 49, Nz=nz)), "fp64")
    gx, gz = 3 * nx // 2, 3 * nz // 2
    rng = np.random.default_rng(5)
    for bad in (np.nan, np.inf, -np.inf):
        phys = rng.normal(size=(3, gz, gx))
        phys[1, 10, 7] = bad
        spec = rng.normal(size=(3, nz, nx // 2 + 1)) + 0j
        spec[1, 4, 3] = bad
        d_spec, d_phys = torch.from_numpy(spec).cuda(), torch.from_numpy(phys).cuda()
        o_phys, o_spec = torch.zeros_like(d_phys), torch.zeros_like(d_spec)
        torch.cuda.synchronize()
        g.four_to_phys(d_spec.data_ptr(), o_phys.data_ptr(), 3)
        g.phys_to_four(d_phys.data_ptr(), o_spec.data_ptr(), 3)
        g.synchronize()
        for got in (o_phys.cpu().numpy(), o_spec.cpu().numpy()):
            assert np.isfinite(got[0]).all() and np.isfinite(got[2]).all()
            assert np.isnan(got[1]).all()
    g.close()
