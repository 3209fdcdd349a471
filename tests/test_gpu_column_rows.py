"""Column transforms of the FP32 form over every height they have (256 to
32768), where few rows of a plane are in the occupancy mask and where most
are, with 1 and 4 pols, image widths that fill the last column tile and that
do not, and one plane-pol or several for a thread block: against the FP64
form, itself held to 1e-10 against direct sums, at the FP32 bar of 1e-5."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(x, dtype):
    return torch.from_numpy(numpy.ascontiguousarray(x)).to("cuda", dtype)


@pytest.mark.parametrize("ny", [128, 256, 512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("nx,npol", [(64, 1), (300, 4)])
@pytest.mark.parametrize("uvscale", [30000.0, 1500.0])
def test_columns_follow_the_occupied_rows(ny, nx, npol, uvscale):
    from rascil_gb300 import wgridder
    c = random_problem(seed=83, nrow=700, nchan=2, npix=8, pixsize=4e-5, uvscale=uvscale,
                       wscale=2500.0, npol=npol)
    img = numpy.random.default_rng(4).normal(size=(npol, nx, ny))

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

    dirty, vis, info, status = both("fp32", "columns", 1e-5, planes_per_batch=5)
    assert info["fft_mode"] == 2 and info["ngrid_y"] == 2 * ny and status == 0
    ref_dirty, ref_vis, _, _ = both("fp64", "auto", 1e-12)
    assert rel_rms(dirty, ref_dirty) < 1e-5
    assert rel_rms(vis, ref_vis) < 1e-5
