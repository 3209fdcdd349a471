"""The FP32 gridder at a support of 9 cells (three support rows of a warp
at a time), with and without w-stacking, 1, 2 and 4 pols, even and odd tiles,
and tiles dense enough for the shared sub-grid: against the FP64 form, itself
held to 1e-10 against direct sums, at the FP32 bar of 1e-5."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(x, dtype):
    return torch.from_numpy(numpy.ascontiguousarray(x)).to("cuda", dtype)


@pytest.mark.parametrize("npol", [1, 2, 4])
@pytest.mark.parametrize("tile", [32, 20, 27])
@pytest.mark.parametrize("do_w", [True, False])
def test_three_rows_at_a_time(npol, tile, do_w):
    from rascil_gb300 import wgridder
    npix = 96
    c = random_problem(seed=47, nrow=5000, nchan=2, npix=npix, wscale=60.0, npol=npol)
    u, f = _dev(c["uvw"], torch.float64), _dev(c["freq"], torch.float64)

    def dirty(precision, eps, **kw):
        cdt = torch.complex128 if precision == "fp64" else torch.complex64
        p = wgridder.Plan(u, f, npix, npix, c["pixsize"], c["pixsize"], eps, do_w, npol=npol,
                          precision=precision, **kw)
        d = p.ms2dirty(_dev(c["ms"], cdt)).double().cpu().numpy()
        info = p.info
        p.close()
        return d, info

    got, info = dirty("fp32", 1e-5, sigma=1.5, tile=tile)
    assert info["support"] == 9 and info["tile"] == tile
    ref, _ = dirty("fp64", 1e-12)
    assert rel_rms(got, ref) < 1e-5
