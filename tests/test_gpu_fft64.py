"""FP64 transforms of the library (k_fft64) over every line length they have, along
rows and along columns, images that fill the middle half of the grid and
ragged ones (a column tile that is not full, padded grids), one and several
batches of w-planes, with and without w-stacking: against the same plan
through cuFFT.  Both are within epsilon of the direct sums (1e-12 here;
tests/test_gpu_fp64.py checks that), so they agree to 2 epsilon, and to the
rounding of the transforms: 5e-12 in all."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(x, dtype):
    return torch.from_numpy(numpy.ascontiguousarray(x)).to("cuda", dtype)


@pytest.mark.parametrize("nx,ny,wstack,uvscale", [
    (64, 64, True, 3000.0), (64, 256, True, 3000.0), (512, 64, True, 30000.0),
    (64, 512, True, 1500.0), (1024, 128, True, 9000.0), (128, 1024, True, 30000.0),
    (2048, 64, True, 30000.0), (64, 2048, True, 30000.0), (256, 256, False, 3000.0),
    (62, 500, True, 30000.0), (1000, 246, False, 30000.0), (486, 2000, True, 30000.0),
])
def test_own_transforms_against_cufft(nx, ny, wstack, uvscale):
    from rascil_gb300 import wgridder
    npol = 2
    c = random_problem(seed=81, nrow=800, nchan=2, npix=8, pixsize=2e-4, uvscale=uvscale,
                       wscale=3000.0, npol=npol)
    img = _dev(numpy.random.default_rng(9).normal(size=(npol, nx, ny)), torch.float64)
    ms = _dev(c["ms"], torch.complex128)

    def both(**kw):
        p = wgridder.Plan(_dev(c["uvw"], torch.float64), _dev(c["freq"], torch.float64), nx, ny,
                          c["pixsize"], c["pixsize"], 1e-12, wstack, npol=npol, precision="fp64",
                          **kw)
        out = p.ms2dirty(ms).cpu().numpy(), p.dirty2ms(img).cpu().numpy(), p.info
        p.close()
        return out

    ref = both(fft_mode="cufft2d", sigma=2.0)
    power = nx & (nx - 1) == 0 and ny & (ny - 1) == 0
    for kw in ({}, dict(planes_per_batch=3)):
        dirty, vis, info = both(sigma=2.0 if power else 0.0, **kw)
        for n in (info["ngrid_x"], info["ngrid_y"]):
            assert n & (n - 1) == 0  # the library's transforms apply
        assert rel_rms(dirty, ref[0]) < 5e-12
        assert rel_rms(vis, ref[1]) < 5e-12
