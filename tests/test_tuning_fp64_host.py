"""The autotuner and the FP64 form's padded grids, on the host: the planner
raises a 486-pixel image's grid sides from 972 to 1024 at epsilon 1e-12, only
at an oversampling of its own choice; the search times that plan, and the
choice it records leads back to it.  FP32 shapes, whose grids are never padded,
keep explicit parameters throughout."""
import pytest


@pytest.fixture
def tuning(tmp_path, monkeypatch):
    from rascil_gb300 import tuning as t
    monkeypatch.setenv("RASCIL_GB300_TUNING", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(t, "_mem", {})
    monkeypatch.setattr(t, "_loaded", [False])
    monkeypatch.setattr(t, "_time", lambda run, cand, repeats: run(cand))
    return t


def _geometry(precision, epsilon, prm):
    from rascil_gb300.wgridder import plan_geometry
    return plan_geometry(486, 486, 5e-4, 5e-4, epsilon, True, -300.0, 300.0, nrows=20000, nchan=2,
                         precision=precision, sigma=prm["sigma"])


def _tune(tuning, precision, epsilon):
    key = tuning.shape_key(486, 486, 5e-4, 1, precision, epsilon, True, 20000, 2)
    own = _geometry(precision, epsilon, tuning.choose(key, 486, 486, 20000, 2))
    start = {"sigma": own["sigma"], "tile": own["tile"], "slab": own["slab"],
             "planes": own["planes_per_batch"]}
    timed = []

    def run(prm):  # stands in for the GPU: power-of-two grids are the fast ones
        g = _geometry(precision, epsilon, prm)
        timed.append(g["ngrid_x"])
        return 1.0 if g["ngrid_x"] & (g["ngrid_x"] - 1) == 0 else 2.0

    best, timings = tuning.autotune(key, run, start=start)
    chosen = tuning.choose(key, 486, 486, 20000, 2)
    return own, best, timings, timed, _geometry(precision, epsilon, chosen)


def test_fp64_search_keeps_the_planners_padded_grid(tuning):
    own, best, timings, timed, got = _tune(tuning, "fp64", 1e-12)
    assert own["ngrid_x"] == 1024 and 1024 in timed and 972 in timed
    assert (got["ngrid_x"], got["sigma"]) == (1024, own["sigma"])
    assert timings[tuning._name(best)] == 1.0


def test_fp32_search_records_an_explicit_oversampling(tuning):
    own, best, timings, timed, got = _tune(tuning, "fp32", 1e-5)
    assert best["sigma"] in tuning.SIGMAS and all("sigma=0" not in name for name in timings)
    assert got["sigma"] == best["sigma"]
