"""FP32 degridder over its dispatch: supports on both sides of the staged range
(up to 7 cells), tiles that can be staged (even, up to 64 cells with the halo)
and that cannot, every polarisation count, chunks below and above the staging
threshold and of several windows of w-planes, batches that cut an item's
planes, supports that wrap round the grid's edges.  Against the FP64 form
with the same support (the same aliasing), so only FP32 rounding differs:
2e-6, the bar for two FP32 forms of one grid."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(x, dtype):
    return torch.from_numpy(numpy.ascontiguousarray(x)).to("cuda", dtype)


@pytest.mark.parametrize("support,npol,wstack,kw", [
    (4, 1, True, {}),
    (4, 4, True, dict(tile=16)),
    (5, 2, True, dict(tile=8, slab=1)),
    (6, 4, True, dict(planes_per_batch=3)),
    (6, 1, False, {}),
    (7, 4, True, {}),
    (7, 1, True, dict(planes_per_batch=5, slab=16)),
    (7, 2, False, dict(tile=30)),
    (7, 1, True, dict(tile=58)),            # 64 cells with the halo: the largest staged for 1 pol
    (7, 4, True, dict(tile=33)),            # odd tile: warp degridder
    (7, 2, True, dict(tile=64)),            # too wide: warp degridder
    (8, 4, True, {}),                       # first support of the warp degridder
    (9, 1, True, dict(planes_per_batch=4)),
])
@pytest.mark.parametrize("npix", [256, 300])
def test_against_the_fp64_form(support, npol, wstack, kw, npix):
    from rascil_gb300 import wgridder
    c = random_problem(seed=91, nrow=900, nchan=2, npix=npix, pixsize=2e-4, uvscale=6000.0,
                       wscale=4000.0, npol=npol)
    # dense buckets: one at a random place, one around the origin (all four corners of the grid)
    c["uvw"][100:400] = c["uvw"][100] + 0.01 * c["uvw"][100:400]
    c["uvw"][400:700] = 0.01 * c["uvw"][400:700]
    weight = 1.0 + numpy.random.default_rng(3).uniform(size=c["wgt"].shape)

    def predict(precision, **more):
        rdt = torch.float64 if precision == "fp64" else torch.float32
        p = wgridder.Plan(_dev(c["uvw"], torch.float64), _dev(c["freq"], torch.float64), npix,
                          npix, c["pixsize"], c["pixsize"], 1e-3, wstack, npol=npol,
                          precision=precision, sigma=2.0, support=support, **more)
        vis = p.dirty2ms(_dev(c["img"], rdt), wgt=_dev(weight, rdt)).cpu().numpy()
        assert p.info["support"] == support and p.device_status() == 0
        p.close()
        return vis

    got = predict("fp32", **kw)
    ref = predict("fp64", fft_mode="cufft2d")
    assert rel_rms(got, ref) < 2e-6


def test_predictions_do_not_depend_on_the_order_of_the_sort():
    """Which items of a bucket share a chunk varies from bind to bind; the
    predictions of one plan do not, bit for bit."""
    from rascil_gb300 import wgridder
    c = random_problem(seed=92, nrow=1500, nchan=3, npix=256, pixsize=2e-4, uvscale=4000.0,
                       wscale=4000.0, npol=4)
    c["uvw"][300:1200] *= 0.01  # buckets of several chunks with short last ones
    img = _dev(c["img"], torch.float32)
    first = None
    for _ in range(6):
        p = wgridder.Plan(_dev(c["uvw"], torch.float64), _dev(c["freq"], torch.float64), 256, 256,
                          c["pixsize"], c["pixsize"], 1e-5, True, npol=4, precision="fp32",
                          sigma=2.0, planes_per_batch=5)
        vis = p.dirty2ms(img).cpu().numpy()
        p.close()
        first = vis if first is None else first
        numpy.testing.assert_array_equal(vis, first)
