"""The FP64 form's w-screens (PlaneScreen<double>, rascil_gb300/csrc/gb_internal.cuh)
against extended precision.

A screen is exp(2 pi i (a + j d)) for the 64-bit phases a and d in turns.  The
bound is what evaluating it directly costs: the phase rounded to a double (up
to 2^-55 of a turn where it is near a half: 1.7e-16 radians, half of that rms
where it is not) and two values rounded (7.9e-17 at most together), so 2.5e-16
at most and 1.0e-16 rms over phases spread evenly."""
import ctypes
import os
import subprocess

import numpy
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "gb_internal.cuh"
__global__ void screens(const unsigned long long *ad, int n, int nb, double2 *out) {
  const double2 *tab = gb::screen_table<double>();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    gb::PlaneScreen<double> ps(tab);
    ps.pt.a = ad[2 * i];
    ps.pt.d = ad[2 * i + 1];
    for (int j = 0; j < nb; ++j) {
      ps.plane(j);
      out[(size_t)i * nb + j] = make_double2(ps.c, ps.s);
    }
  }
}
extern "C" int run(const unsigned long long *ad, int n, int nb, double2 *out) {
  screens<<<32, 256>>>(ad, n, nb, out);
  return (int)cudaDeviceSynchronize();
}
"""


def test_fp64_screens(tmp_path):
    from rascil_gb300 import build
    src, lib = tmp_path / "screens.cu", tmp_path / "screens.so"
    src.write_text(SOURCE)
    csrc = os.path.join(build.HERE, "csrc")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", csrc,
                    "-I", os.path.join(build.HERE, "..", "include"), "-shared", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    n, nb = 20000, 21
    rng = numpy.random.default_rng(17)
    ad = rng.integers(0, 2 ** 64, (n, 2), dtype=numpy.uint64)
    # phases at and next to the table's points and half way between them, and all ones
    edge = numpy.array([0, 1, 2 ** 55 - 1, 2 ** 55, 2 ** 55 + 1, 2 ** 56, 2 ** 61, 2 ** 62, 2 ** 63,
                        2 ** 64 - 2 ** 55 - 1, 2 ** 64 - 2 ** 55, 2 ** 64 - 1], dtype=numpy.uint64)
    ad[:len(edge), 0] = edge
    ad[:len(edge), 1] = 0
    a = torch.from_numpy(ad.view(numpy.int64)).cuda()
    out = torch.empty((n, nb), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    so = ctypes.CDLL(str(lib))
    assert so.run(ctypes.c_void_p(a.data_ptr()), n, nb, ctypes.c_void_p(out.data_ptr())) == 0
    got = out.cpu().numpy()
    with numpy.errstate(over="ignore"):
        ph = ad[:, :1] + numpy.arange(nb, dtype=numpy.uint64) * ad[:, 1:]
    L = numpy.longdouble
    turns = ph.view(numpy.int64).astype(L) / L(2) ** 64  # in [-1/2, 1/2), exact
    angle = turns * (L(2) * L("3.14159265358979323846264338327950288"))
    err = numpy.hypot((got.real - numpy.cos(angle)).astype(float),
                      (got.imag - numpy.sin(angle)).astype(float))
    assert err.max() < 2.5e-16
    assert numpy.sqrt(numpy.mean(err ** 2)) < 1.0e-16
