"""Rounding error of the FP32 row transforms (k_rows) inside a prediction:
against the FP64 form with the same grid and support, which has the same
aliasing, so that what is left is the FP32 form's rounding.

The bounds are what these problems gave (mean of eight) when every factor
w^(8 a t) of the first pass was a table value and the transforms ran in scalar
arithmetic, plus 0.2 %; a prediction of given inputs is the same in every run.
Factors formed as powers of w^(8 t) gave 0.4 to 1.0 % more."""
import numpy
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,before", [(2048, 5.9422e-7), (4096, 5.9673e-7), (8192, 5.9323e-7)])
def test_no_more_than_scalar_transforms_with_table_factors(nx, before):
    from rascil_gb300 import wgridder
    ny, n, pix = 128, 4000, 0.05 / nx
    errors = []
    for seed in range(8):
        rng = numpy.random.default_rng(seed)
        uvw = numpy.stack([rng.uniform(-.45, .45, n) / pix, rng.uniform(-.45, .45, n) / pix,
                           rng.uniform(0, 4000., n)], 1)
        uvw = torch.from_numpy(uvw).cuda()
        freq = torch.full((1,), 299792458.0, dtype=torch.float64, device="cuda")
        img = torch.from_numpy(rng.normal(size=(1, ny, nx)).astype(numpy.float32)).cuda()
        vis = {}
        for precision, mode in (("fp64", "cufft2d"), ("fp32", "columns")):
            p = wgridder.Plan(uvw, freq, nx, ny, pix, pix, 1e-5, True, precision=precision,
                              fft_mode=mode, sigma=2.0, support=7)
            assert p.info["ngrid_x"] == 2 * nx and p.info["own_rows"] == (precision == "fp32")
            vis[precision] = p.dirty2ms(img.to(p.real_dtype), layout="yx").to(torch.complex128)
            p.close()
        errors.append(float((vis["fp32"] - vis["fp64"]).norm() / vis["fp64"].norm()))
    assert numpy.mean(errors) < 1.002 * before
