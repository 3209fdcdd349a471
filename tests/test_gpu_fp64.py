"""FP64 tile kernels (k_grid64, k_degrid64) at the edges of their ranges.

Against the oracle's FP64 direct sums: every support width class (cells per
lane of the degridder), every polarisation count, non-default tiles and
slabs, w-planes split over several batches, buckets of one item and of more
than a chunk.  The tolerance is the requested epsilon, which the kernel
table guarantees for the aliasing, with a floor of 2e-13 for the rounding of
the transforms.
"""
import numpy
import pytest

from cases import random_problem, rel_rms
from oracle import dft

pytestmark = pytest.mark.gpu


def _plan(c, npol, eps, wstack=True, **kw):
    import torch
    from rascil_gb300 import wgridder
    u = torch.from_numpy(c["uvw"]).cuda()
    f = torch.from_numpy(c["freq"]).cuda()
    return wgridder.Plan(u, f, c["npix"], c["npix"], c["pixsize"], c["pixsize"], eps, wstack,
                         npol=npol, precision="fp64", **kw)


@pytest.mark.parametrize("eps,npol,wstack,kw", [
    (3e-3, 1, True, {}),                                   # W 4: one cell per lane
    (1e-4, 4, True, dict(tile=4, slab=1)),                 # smallest tile and slab
    (1e-6, 2, True, dict(planes_per_batch=1)),             # every plane its own batch
    (1e-8, 1, True, dict(planes_per_batch=5, slab=3)),     # items across batches
    (1e-10, 4, True, dict(planes_per_batch=7)),
    (1e-12, 1, True, dict(tile=33, slab=128)),             # wide tile, one slab
    (8e-14, 2, True, {}),                                  # W 16
    (8e-14, 1, False, dict(tile=96)),                      # no w-stacking, 111 x 111 sub-grid
])
def test_both_directions_against_direct_sums(eps, npol, wstack, kw):
    import torch
    c = random_problem(seed=3, nrow=300, nchan=2, npix=64, npol=npol)
    # a dense clump: one bucket of several chunks, and rows that are alone
    c["uvw"][100:250] = c["uvw"][100] + 1e-3 * c["uvw"][100:250]
    plan = _plan(c, npol, eps, wstack, **kw)
    ms, wgt = torch.from_numpy(c["ms"]).cuda(), torch.from_numpy(c["wgt"]).cuda()
    dirty = plan.ms2dirty(ms, wgt=wgt, layout="xy").cpu().numpy()
    img = torch.from_numpy(c["img"]).cuda()
    vis = plan.dirty2ms(img, layout="xy").cpu().numpy()
    tol = max(eps, 2e-13)
    for p in range(npol):
        ref = dft.ms2dirty_dft(c["uvw"], c["freq"], c["ms"][..., p], c["wgt"][..., p], c["npix"],
                               c["npix"], c["pixsize"], c["pixsize"], wstack)
        assert rel_rms(dirty[p], ref) < tol
        ref = dft.dirty2ms_dft(c["uvw"], c["freq"], c["img"][p], None, c["pixsize"],
                               c["pixsize"], wstack)
        assert rel_rms(vis[..., p], ref) < tol


@pytest.mark.parametrize("power", [-880, -300, 300, 900])
def test_magnitudes(power):
    """The gridder's fixed point follows the data's magnitude: scaling the
    visibilities by a power of two scales the image exactly (to the order of
    the grid's atomic additions)."""
    import torch
    c = random_problem(seed=4, nrow=200, nchan=1, npix=32)
    plan = _plan(c, 1, 1e-10)
    ms = torch.from_numpy(c["ms"]).cuda()
    one = plan.ms2dirty(ms, layout="yx").cpu().numpy()
    scaled = plan.ms2dirty(ms * 2.0 ** power, layout="yx").cpu().numpy()
    assert rel_rms(scaled * 2.0 ** -power, one) < 1e-14


@pytest.mark.parametrize("bad", [numpy.nan, numpy.inf, -numpy.inf])
def test_non_finite_values_reach_their_polarisation_only(bad):
    import torch
    c = random_problem(seed=5, nrow=200, nchan=1, npix=32, npol=2)
    plan = _plan(c, 2, 1e-10)
    clean = plan.ms2dirty(torch.from_numpy(c["ms"]).cuda(), layout="yx").cpu().numpy()
    c["ms"][17, 0, 1] = bad
    got = plan.ms2dirty(torch.from_numpy(c["ms"]).cuda(), layout="yx").cpu().numpy()
    assert not numpy.isfinite(got[1]).any()
    assert rel_rms(got[0], clean[0]) < 1e-14


@pytest.mark.parametrize("precision,eps,kw", [
    ("fp64", 8e-14, [{}, dict(support=4)]),
    ("fp32", 1e-5, [dict(tile=48), dict(tile=4)]),
])
def test_plans_of_other_shared_memory_do_not_disturb_each_other(precision, eps, kw):
    """A kernel's shared-memory opt-in belongs to the kernel: a plan that needs
    little, made later, must not take it from one that needs more."""
    import torch
    from rascil_gb300 import wgridder
    c = random_problem(seed=6, nrow=200, nchan=1, npix=64)
    u = torch.from_numpy(c["uvw"]).cuda()
    f = torch.from_numpy(c["freq"]).cuda()
    ms = torch.from_numpy(c["ms"]).cuda()
    plans = []
    for extra in kw:
        p = wgridder.Plan(u, f, 64, 64, c["pixsize"], c["pixsize"], eps, True, npol=1,
                          precision=precision, sigma=2.0, **extra)
        plans.append((p, p.ms2dirty(ms.to(p.complex_dtype), layout="yx").clone()))
    for p, before in plans:
        again = p.ms2dirty(ms.to(p.complex_dtype), layout="yx")
        assert rel_rms(again.cpu().numpy(), before.cpu().numpy()) < 1e-6
