"""Work chunks (FP64: 8 to 64 items) and the parts of them that the FP32 gridder
takes (64 to 256 items) shorten with the item count.  Item counts on both sides of each step, in clumped and in scattered
buckets: the FP64 form against the oracle's direct sums at the requested
epsilon, the FP32 form against the FP64 form at the FP32 bar of 1e-5."""
import numpy
import pytest

from oracle import dft
from tests.cases import random_problem, rel_rms

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _problem(nrow, npix, npol):
    c = random_problem(seed=61, nrow=nrow, nchan=1, npix=npix, wscale=200.0, npol=npol)
    c["uvw"][: nrow // 3] *= 0.02  # a dense clump
    return c


def _both(c, npol, precision, eps, **kw):
    from rascil_gb300 import wgridder
    rdt, cdt = ((torch.float64, torch.complex128) if precision == "fp64" else
                (torch.float32, torch.complex64))
    p = wgridder.Plan(torch.from_numpy(c["uvw"]).cuda(), torch.from_numpy(c["freq"]).cuda(),
                      c["npix"], c["npix"], c["pixsize"], c["pixsize"], eps, True, npol=npol,
                      precision=precision, **kw)
    dirty = p.ms2dirty(torch.from_numpy(c["ms"]).to("cuda", cdt), layout="xy")
    vis = p.dirty2ms(torch.from_numpy(c["img"]).to("cuda", rdt), layout="xy")
    p.close()
    return dirty.double().cpu().numpy(), vis.cpu().numpy()


@pytest.mark.parametrize("nrow", [9, 16383, 16384, 32768, 65535, 65536])
def test_fp64(nrow):
    c = _problem(nrow, 16, 1)
    dirty, vis = _both(c, 1, "fp64", 1e-10)
    ref = dft.ms2dirty_dft(c["uvw"], c["freq"], c["ms"][..., 0], None, 16, 16, c["pixsize"],
                           c["pixsize"], True)
    assert rel_rms(dirty[0], ref) < 1e-10
    ref = dft.dirty2ms_dft(c["uvw"], c["freq"], c["img"][0], None, c["pixsize"], c["pixsize"],
                           True)
    assert rel_rms(vis[..., 0], ref) < 1e-10


@pytest.mark.parametrize("nrow", [65, 65535, 65536, 131071, 131072])
@pytest.mark.parametrize("npol", [1, 4])
def test_fp32(nrow, npol):
    c = _problem(nrow, 64, npol)
    got = _both(c, npol, "fp32", 1e-5, sigma=2.0)
    ref = _both(c, npol, "fp64", 1e-12)
    assert rel_rms(got[0], ref[0]) < 1e-5
    assert rel_rms(got[1], ref[1]) < 1e-5
