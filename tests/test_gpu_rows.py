"""Row transforms of the FP32 form (k_rows) over every width they have, with
images that fill the middle half of the row and ragged ones, and with
visibilities in most bins of the occupancy mask (more than the stage holds)
or in few: against the FP64 GPU form, itself held to 1e-10 against direct
sums, at the FP32 bar of 1e-5, and against the batched cuFFT transforms at
2e-6 (two FP32 forms of the same grid)."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(x, dtype):
    return torch.from_numpy(numpy.ascontiguousarray(x)).to("cuda", dtype)


# grid widths 512 ... 16384; the second of a pair is ragged (no width of 512 has one)
@pytest.mark.parametrize("nx", [256, 512, 508, 1024, 1020, 2048, 2044, 4096, 4092, 8192, 8188])
@pytest.mark.parametrize("uvscale", [30000.0, 2500.0])
def test_rows_follow_the_occupied_bins(nx, uvscale):
    from rascil_gb300 import wgridder
    ny, npol = 128, 2
    c = random_problem(seed=71, nrow=1200, nchan=2, npix=8, pixsize=5e-5, uvscale=uvscale,
                       wscale=3000.0, npol=npol)
    img = numpy.random.default_rng(9).normal(size=(npol, nx, ny))

    def both(precision, mode, eps, **kw):
        rdt, cdt = ((torch.float64, torch.complex128) if precision == "fp64" else
                    (torch.float32, torch.complex64))
        p = wgridder.Plan(_dev(c["uvw"], torch.float64), _dev(c["freq"], torch.float64), nx, ny,
                          c["pixsize"], c["pixsize"], eps, True, npol=npol, precision=precision,
                          fft_mode=mode, sigma=2.0, **kw)
        dirty = p.ms2dirty(_dev(c["ms"], cdt)).double().cpu().numpy()
        vis = p.dirty2ms(_dev(img, rdt)).cpu().numpy()
        info, status = p.info, p.device_status()
        p.close()
        return dirty, vis, info, status

    dirty, vis, info, status = both("fp32", "columns", 1e-5, planes_per_batch=3)
    assert info["own_rows"] == 1 and info["ngrid_x"] >= 2 * nx and status == 0
    ref_dirty, ref_vis, _, _ = both("fp64", "auto", 1e-12)
    assert rel_rms(dirty, ref_dirty) < 1e-5
    assert rel_rms(vis, ref_vis) < 1e-5
    # the same grids through cuFFT
    two_dirty, two_vis, two, _ = both("fp32", "cufft2d", 1e-5)
    assert two["fft_mode"] == 1 and two["ngrid_x"] == info["ngrid_x"]
    assert rel_rms(dirty, two_dirty) < 2e-6
    assert rel_rms(vis, two_vis) < 2e-6
