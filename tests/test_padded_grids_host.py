"""The planner raises the FP64 form's grid sides to powers of two (for the
library's own transforms) only at an oversampling of its own choice and an
epsilon of 1e-9 or below: another grid moves a result by up to epsilon.  Host
only."""
import pytest


def _sides(npix, epsilon, **kw):
    from rascil_gb300.wgridder import plan_geometry
    p = plan_geometry(npix, npix, 5e-4, 5e-4, epsilon, True, -300.0, 300.0, nrows=20000, nchan=2,
                      precision=kw.pop("precision", "fp64"), **kw)
    assert p["ngrid_x"] == p["ngrid_y"]
    return p["ngrid_x"], p["sigma"]


@pytest.mark.parametrize("epsilon,padded", [(1e-12, True), (1e-9, True), (1.01e-9, False),
                                            (1e-6, False)])
def test_only_at_small_epsilon(epsilon, padded):
    side, sigma = _sides(486, epsilon)
    assert sigma == 2.0 and side == (1024 if padded else 972)


def test_not_where_the_caller_fixes_the_oversampling_or_the_form_is_fp32():
    assert _sides(486, 1e-12, sigma=2.0)[0] == 972
    side, sigma = _sides(486, 1e-5, precision="fp32")
    assert side & (side - 1) != 0


def test_not_where_the_larger_grid_costs_more():
    assert _sides(260, 1e-12)[0] == 540  # 1024 has 3.6 times the cells
