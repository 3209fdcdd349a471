"""FP32 gridding with odd tile sides: tile origins are then odd for every other
tile, so the flush may not add two cells with one 16-byte atomic there (and a
pair may straddle the grid's edge)."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [5, 31, 33])
@pytest.mark.parametrize("npol", [1, 4])
def test_invert_with_an_odd_tile(tile, npol):
    from rascil_gb300 import wgridder
    c = random_problem(seed=95, nrow=600, nchan=2, npix=256, pixsize=2e-4, uvscale=5000.0,
                       wscale=3000.0, npol=npol)
    # dense buckets (the sub-grid path), one of them around the grid's corner
    c["uvw"][100:300] = c["uvw"][100] + 0.01 * c["uvw"][100:300]
    c["uvw"][300:500] *= 0.01
    u = torch.from_numpy(c["uvw"]).cuda()
    f = torch.from_numpy(c["freq"]).cuda()
    ms = torch.from_numpy(c["ms"]).to("cuda", torch.complex64)

    def dirty(precision, **kw):
        p = wgridder.Plan(u, f, 256, 256, c["pixsize"], c["pixsize"], 1e-5, True, npol=npol,
                          precision=precision, sigma=2.0, **kw)
        out = p.ms2dirty(ms.to(p.complex_dtype), layout="yx").double().cpu().numpy()
        support = p.info["support"]
        p.close()
        return out, support

    got, support = dirty("fp32", tile=tile)
    ref, _ = dirty("fp64", support=support)
    # the same aliasing in both forms: FP32 rounding only
    assert rel_rms(got, ref) < 2e-6
