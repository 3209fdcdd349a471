"""A plan's results do not depend on what its workspace held before: both
directions on a buffer of 0xFF bytes (a NaN in every float and double) against
the same plan on a zeroed buffer, for every form and transform.

The transforms follow a plan's occupancy mask, so much of the workspace is
never written; whatever reads a cell outside the mask reads these NaN.  The
two bindings do the same operations, only the order of the additions into a
grid cell may differ: a few roundings (1.2e-7 and 2.2e-16) of the grid's
largest terms, up to 30 times as large at the image's edge after the
correction, so 1e-5 and 1e-13 hold for both directions."""
import numpy
import pytest

from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FP64_OWN, FP64_LIB, ROWS, LIB_ROWS, LIB = range(5)


def _problem(nx, ny, npol, pixsize, away, wscale=30000.0):
    """Items all over the uv plane, or with `away` none near u = 0 or v = 0:
    no support then reaches cell (0, 0) of any w-plane, nor its neighbours."""
    c = random_problem(seed=91, nrow=700, nchan=2, npix=8, pixsize=pixsize, npol=npol,
                       uvscale=0.45 / pixsize / 0.467, wscale=wscale)
    if away:
        rng = numpy.random.default_rng(92)
        c["uvw"][:, :2] = (rng.choice([-1.0, 1.0], (700, 2)) * rng.uniform(0.2, 0.4, (700, 2))
                           / pixsize / 0.467)
    dev = lambda x: torch.from_numpy(numpy.ascontiguousarray(x)).cuda()
    img = numpy.random.default_rng(93).normal(size=(npol, nx, ny))
    return dev(c["uvw"]), dev(c["freq"]), dev(c["ms"]), dev(img)


def _bind(plan, byte):
    plan.bind(torch.full((plan.workspace_bytes,), byte, dtype=torch.uint8, device="cuda"))


def _check_transform(info, transform, nx, ny):
    gx, gy = info["ngrid_x"], info["ngrid_y"]
    power = gx & (gx - 1) == 0 and gy & (gy - 1) == 0
    if transform in (ROWS, LIB_ROWS):
        assert info["fft_mode"] == 2 and info["own_rows"] == (transform == ROWS)
    else:
        assert info["fft_mode"] == 1
    if transform == FP64_OWN:  # what sends a plan to the library's own transforms
        assert power and min(gx, gy) >= 128 and gx >= 2 * nx and gy >= 2 * ny


@pytest.mark.parametrize("away", [False, True])
@pytest.mark.parametrize("precision,transform,nx,ny,npol,eps,wstack,kw", [
    ("fp64", FP64_OWN, 256, 256, 1, 1e-12, True, {}),
    ("fp64", FP64_OWN, 512, 128, 2, 1e-10, True, dict(planes_per_batch=5)),
    ("fp64", FP64_OWN, 128, 1024, 4, 1e-8, True, dict(sigma=2.0)),
    ("fp64", FP64_OWN, 64, 64, 1, 1e-3, True, dict(sigma=2.0, tile=4)),
    ("fp64", FP64_OWN, 486, 250, 1, 1e-11, True, {}),
    ("fp64", FP64_OWN, 256, 512, 2, 1e-9, False, dict(sigma=2.0)),
    ("fp64", FP64_LIB, 256, 256, 1, 1e-12, True, dict(fft_mode="cufft2d")),
    ("fp64", FP64_LIB, 150, 200, 4, 1e-6, False, dict(sigma=1.5)),
    ("fp32", ROWS, 256, 256, 4, 1e-5, True, dict(sigma=2.0)),
    ("fp32", ROWS, 508, 512, 1, 1e-5, True, dict(sigma=2.0, support=7, planes_per_batch=3)),
    ("fp32", LIB_ROWS, 500, 512, 1, 1e-5, True, dict(sigma=2.0, support=7, planes_per_batch=3)),
    ("fp32", ROWS, 1024, 128, 2, 1e-3, True, dict(sigma=2.0, tile=16)),
    ("fp32", ROWS, 2048, 256, 1, 1e-5, True, dict(sigma=2.0)),
    ("fp32", ROWS, 256, 1024, 1, 1e-5, False, dict(sigma=2.0)),
    ("fp32", LIB_ROWS, 200, 256, 2, 1e-5, True, dict(sigma=2.0)),
    ("fp32", LIB, 256, 256, 1, 1e-5, True, dict(sigma=2.0, fft_mode="cufft2d")),
    ("fp32", LIB, 150, 170, 2, 1e-4, False, {}),
    ("fp32", LIB, 150, 170, 4, 1e-5, True, dict(sigma=1.5, tile=27)),
])
def test_results_do_not_depend_on_the_buffer(precision, transform, nx, ny, npol, eps, wstack, kw,
                                             away):
    from rascil_gb300 import wgridder
    pixsize = 2e-4
    uvw, freq, ms, img = _problem(nx, ny, npol, pixsize, away)
    plan = wgridder.Plan(uvw, freq, nx, ny, pixsize, pixsize, eps, wstack, npol=npol,
                         precision=precision, bind=False, **kw)
    _check_transform(plan.info, transform, nx, ny)
    ms, img = ms.to(plan.complex_dtype), img.to(plan.real_dtype)
    got = {}
    for byte in (0x00, 0xFF):
        # each direction first on its own buffer, then after the other
        _bind(plan, byte)
        vis = plan.dirty2ms(img).cpu().numpy()
        after = plan.ms2dirty(ms).cpu().numpy()
        _bind(plan, byte)
        dirty = plan.ms2dirty(ms).cpu().numpy()
        got[byte] = (vis, after, dirty, plan.dirty2ms(img).cpu().numpy())
    plan.close()
    tol = 1e-13 if precision == "fp64" else 1e-5
    for clean, stale in zip(got[0x00], got[0xFF]):
        assert numpy.isfinite(clean).all()
        bad = numpy.count_nonzero(~numpy.isfinite(stale))
        assert bad == 0, "%d of %d values not finite" % (bad, stale.size)
        assert rel_rms(stale, clean) < tol


@pytest.mark.parametrize("nx,ny,eps,kw", [
    (256, 256, 1e-12, {}), (512, 128, 1e-10, dict(planes_per_batch=4)),
    (486, 250, 1e-11, {}), (64, 64, 1e-3, dict(sigma=2.0, tile=4)),
])
@pytest.mark.parametrize("bad", [numpy.nan, numpy.inf])
def test_non_finite_values_through_own_transforms(nx, ny, eps, kw, bad):
    """A non-finite visibility makes its polarisation's whole image non-finite
    also where no visibility reaches the grid's first cells, and leaves nothing
    behind: predictions of the same plan stay as they were."""
    from rascil_gb300 import wgridder
    pixsize = 2e-4
    uvw, freq, ms, img = _problem(nx, ny, 2, pixsize, True)
    plan = wgridder.Plan(uvw, freq, nx, ny, pixsize, pixsize, eps, True, npol=2,
                         precision="fp64", **kw)
    _check_transform(plan.info, FP64_OWN, nx, ny)
    before = plan.dirty2ms(img).cpu().numpy()
    clean = plan.ms2dirty(ms).cpu().numpy()
    ms[317, 1, 1] = bad
    dirty = plan.ms2dirty(ms).cpu().numpy()
    after = plan.dirty2ms(img).cpu().numpy()
    plan.close()
    assert not numpy.isfinite(dirty[1]).any()
    assert rel_rms(dirty[0], clean[0]) < 1e-13
    assert numpy.isfinite(after).all() and rel_rms(after, before) < 1e-13
