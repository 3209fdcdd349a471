"""The work whose speed this framework is measured by.

Each case is one call (or the few calls that go together) that a user of the
framework makes, through its public entry points, on a synthetic observation
of one of the array configurations of ``rascil_gb300.simulation``.  Sizes run
from a snapshot of a small array on a 64-pixel image to a whole field of four
polarisations on 8192 x 8192 pixels.  Calls at the level of a plan hold their
data on the device, as a pipeline on the GPU does; ``invert_ng``,
``predict_ng`` and ``weight_visibility`` take host data, as RASCIL calls them.
"""
import math

import numpy
import torch

DEVICE = "cuda"
C_LIGHT = 299792458.0

# linear (XX, XY, YX, YY) -> (I, Q, U, V) and back: the polarisation matrices
# of a four-polarisation pipeline (TMS 4.58)
LINEAR_TO_IQUV = 0.5 * numpy.array([[1, 0, 0, 1], [1, 0, 0, -1], [0, 1, 1, 0], [0, -1j, 1j, 0]])
IQUV_TO_LINEAR = numpy.array([[1, 1, 0, 0], [0, 0, 1, 1j], [0, 0, 1, -1j], [1, -1, 0, 0]],
                             dtype=complex)


def listed():
    return [
        # A script's ducc0-style calls on a short snapshot of a small array:
        # plan, sort, grid and transform per call, where launches, host work
        # and allocations count more than the data.
        dict(name="ducc0-calls-small", kind="oneshot", config="small-array", nants=32, ntimes=2,
             nchan=2, npixel=256, npol=1, precision="fp32", epsilon=1e-5, wstack=True),
        # RASCIL's own round trip with its defaults (double precision, epsilon
        # 1e-12, host data) on the small-array configuration: predict_ng of a
        # sky model, then invert_ng of what was predicted.
        dict(name="ng-round-trip-default", kind="ng", config="small-array", nants=64, ntimes=64,
             nchan=1, npixel=512, npol=1, precision="fp64", epsilon=1e-12, wstack=True),
        # Double-precision imaging of four polarisations with flags and
        # weights, an image size that is no power of two.
        dict(name="invert-fp64-iquv", kind="invert", config="small-array", nants=64, ntimes=24,
             nchan=3, npixel=486, npol=4, precision="fp64", epsilon=1e-10, wstack=True),
        # Double-precision prediction of a component model for calibration.
        dict(name="predict-fp64", kind="predict", config="gain-solve", nants=128, ntimes=16,
             nchan=4, npixel=1024, npol=1, precision="fp64", epsilon=1e-8, wstack=True),
        # Imaging an observation of a low-frequency array, all baselines, four
        # polarisations: the direction that a major cycle runs per iteration.
        dict(name="invert-low-iquv", kind="invert", config="low-like", nants=512, ntimes=16,
             nchan=16, npixel=4096, npol=4, precision="fp32", epsilon=1e-5, wstack=True),
        # The other direction of the same major cycle.
        dict(name="predict-low-iquv", kind="predict", config="low-like", nants=512, ntimes=16,
             nchan=16, npixel=4096, npol=4, precision="fp32", epsilon=1e-5, wstack=True),
        # A new block of a dish array's data, wide image: the plan (sort and
        # tables) with one invert and one predict, nothing to reuse.
        dict(name="step-mid-wide", kind="step", config="mid-like", nants=197, ntimes=8,
             nchan=64, npixel=8192, npol=4, precision="fp32", epsilon=1e-5, wstack=True),
        # A core-station snapshot imaged without w-stacking: two polarisations,
        # ragged sizes, looser accuracy.
        dict(name="invert-2d-ragged", kind="invert", config="low-like", nants=100, ntimes=9,
             nchan=5, npixel=1250, npol=2, precision="fp32", epsilon=1e-4, wstack=False),
        # One gradient step of a joint sky and gain solve: differentiable
        # predict, per-antenna gains, backward to both.
        dict(name="gain-solve-step", kind="gains", config="gain-solve", nants=128, ntimes=64,
             nchan=8, npixel=2048, npol=1, precision="fp32", epsilon=1e-5, wstack=True),
        # A list of snapshots of uneven size, wide fields and few visibilities
        # each, solved as one program.
        dict(name="snapshot-batch", kind="batch", nsnap=12, shapes=3, maxvis=1000000,
             precision="fp32", epsilon=1e-5),
        # Predicting a bright-source list exactly (no image).
        dict(name="component-dft", kind="dft", config="gain-solve", nants=128, ntimes=8, nchan=8,
             npol=1, ncomp=200, precision="fp64", exact=True),
        # Uniform imaging weights before a first image, host data.
        dict(name="uniform-weights", kind="weights", config="low-like", nants=200, ntimes=4,
             nchan=4, npixel=4096, npol=4, weighting="uniform"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """An image side: even (the gridder's rule), often a power of two."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.4:
        return 1 << int(round(math.log2(n)))
    return max(lo, min(hi, n + n % 2))


def draw(rng):
    kind = rng.choice(["oneshot", "ng", "fp64", "fp64", "fp32", "fp32", "fp32", "step", "gains",
                       "batch", "dft", "weights"])
    if kind in ("oneshot", "ng"):
        fp32 = kind == "oneshot" and rng.random() < 0.6
        return dict(kind=kind, config="small-array", nants=_log(rng, 12, 64),
                    ntimes=_log(rng, 1, 16 if kind == "oneshot" else 64),
                    nchan=1 if kind == "ng" else _log(rng, 1, 4), npixel=_side(rng, 64, 512),
                    npol=1, precision="fp32" if fp32 else "fp64",
                    epsilon=rng.choice([1e-3, 1e-4, 1e-5]) if fp32 else
                    rng.choice([1e-6, 1e-9, 1e-12]),
                    wstack=kind == "ng" or rng.random() < 0.8)
    if kind == "fp64":
        return dict(kind=rng.choice(["invert", "predict"]),
                    config=rng.choice(["small-array", "gain-solve"]), nants=_log(rng, 16, 64),
                    ntimes=_log(rng, 2, 24), nchan=_log(rng, 1, 3), npixel=_side(rng, 128, 512),
                    npol=rng.choice([1, 2, 4]), precision="fp64",
                    epsilon=rng.choice([1e-6, 1e-8, 1e-10, 1e-12]), wstack=rng.random() < 0.8)
    if kind == "fp32":
        return dict(kind=rng.choice(["invert", "predict"]),
                    config=rng.choice(["small-array", "low-like", "low-like", "gain-solve"]),
                    nants=_log(rng, 48, 512), ntimes=_log(rng, 1, 16), nchan=_log(rng, 1, 16),
                    npixel=min(_side(rng, 128, 4096), 4096), npol=rng.choice([1, 2, 4]),
                    precision="fp32", epsilon=rng.choice([1e-3, 1e-4, 1e-5, 1e-5]),
                    wstack=rng.random() < 0.85)
    if kind == "step":
        config = rng.choice(["low-like", "mid-like"])
        return dict(kind=kind, config=config, nants=_log(rng, 48, 197), ntimes=_log(rng, 1, 8),
                    nchan=_log(rng, 1, 32), npixel=_side(rng, 256, 4096),
                    npol=rng.choice([1, 4]), precision="fp32", epsilon=1e-5, wstack=True)
    if kind == "gains":
        return dict(kind=kind, config="gain-solve", nants=_log(rng, 24, 128),
                    ntimes=_log(rng, 4, 64), nchan=_log(rng, 1, 8), npixel=_side(rng, 256, 2048),
                    npol=1, precision="fp32", epsilon=1e-5, wstack=True)
    if kind == "batch":
        return dict(kind=kind, nsnap=rng.randint(3, 11), shapes=rng.randint(4, 1000),
                    maxvis=_log(rng, 50000, 1000000), precision="fp32", epsilon=1e-5)
    if kind == "dft":
        fp64 = rng.random() < 0.5
        return dict(kind=kind, config="gain-solve", nants=_log(rng, 16, 128),
                    ntimes=_log(rng, 1, 8), nchan=_log(rng, 1, 8), npol=rng.choice([1, 2, 4]),
                    ncomp=_log(rng, 5, 150), precision="fp64" if fp64 else "fp32",
                    exact=fp64 or rng.random() < 0.3)
    return dict(kind="weights", config="low-like", nants=_log(rng, 24, 200),
                ntimes=_log(rng, 1, 4), nchan=_log(rng, 1, 4), npixel=_side(rng, 3072, 4096),
                npol=rng.choice([1, 2, 4]), weighting=rng.choice(["uniform", "robust", "natural"]))


# ----------------------------------------------------------------------
# observations

def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 13)


def _observation(case, seed):
    """(uvw [rows, 3] numpy, metres, freq, config, declination)."""
    from rascil_gb300.simulation import observation
    uvw, freq, centre, cfg = observation(case["config"], seed=int(seed) % 100003,
                                         ntimes=case["ntimes"], nchan=case["nchan"],
                                         nants=case["nants"])
    return uvw, freq, centre, cfg


def _device_uvw(uvw):
    """uvw as ng.py hands them to the gridder (u and w negated)."""
    u = torch.from_numpy(numpy.ascontiguousarray(uvw.reshape(-1, 3))).to(DEVICE)
    return u * torch.tensor([-1.0, 1.0, -1.0], dtype=torch.float64, device=DEVICE)


def _sky(npixel, cell, npol, seed, nsrc=200):
    """Pixels (x, y) and fluxes [nsrc, npol] of a CLEAN-component model: power
    -law Stokes I inside the inner 80 % of the field, a few per cent polarised."""
    rng = numpy.random.default_rng(int(seed) + 501)
    half = max(1, int(0.4 * npixel))
    x = npixel // 2 + rng.integers(-half, half, nsrc)
    y = npixel // 2 + rng.integers(-half, half, nsrc)
    flux = numpy.zeros((nsrc, npol))
    flux[:, 0] = 0.01 * rng.uniform(size=nsrc) ** -0.7
    for p in range(1, npol):
        flux[:, p] = 0.05 * flux[:, 0] * rng.normal(size=nsrc)
    return x, y, flux


def _model(npixel, cell, npol, seed, dtype, order):
    """The sky as an image: [npol, y, x] or, for order "xy", [npol, x, y]."""
    x, y, flux = _sky(npixel, cell, npol, seed)
    img = torch.zeros((npol, npixel, npixel), dtype=torch.float64, device=DEVICE)
    ix = torch.from_numpy(x).to(DEVICE)
    iy = torch.from_numpy(y).to(DEVICE)
    f = torch.from_numpy(flux).to(DEVICE)
    for p in range(npol):
        img[p].index_put_((ix, iy) if order == "xy" else (iy, ix), f[:, p], accumulate=True)
    return img.to(dtype)


def _noisy_vis(uvw, freq, npol, half_field, seed, dtype):
    """Visibilities [rows, chans, npol]: a few bright sources under noise that
    is several times the faint ones, as a correlator gives them."""
    g = _generator(seed)
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    shape = (uvw.shape[0], freq.shape[0], npol)
    vis = torch.view_as_complex(0.3 * torch.randn(shape + (2,), generator=g, device=DEVICE,
                                                  dtype=real))
    rng = numpy.random.default_rng(int(seed) + 77)
    k = freq / C_LIGHT
    for _ in range(3):
        l, m = (rng.uniform(-0.7, 0.7, 2) * half_field).tolist()
        n1 = math.sqrt(1.0 - l * l - m * m) - 1.0
        turns = (l * uvw[:, 0] + m * uvw[:, 1] - n1 * uvw[:, 2])[:, None] * k
        turns = 2.0 * math.pi * (turns - torch.round(turns))
        wave = torch.polar(torch.full_like(turns, rng.uniform(0.2, 2.0)), -turns).to(dtype)
        vis[:, :, 0] += wave
        if npol == 4:
            vis[:, :, 3] += 0.9 * wave
    return vis


def _weights_and_flags(shape, seed, real):
    """Imaging weights and RASCIL's int64 flags (6 % set)."""
    g = _generator(seed + 1)
    wgt = 0.5 + torch.rand(shape, generator=g, device=DEVICE, dtype=real)
    flags = (torch.rand(shape, generator=g, device=DEVICE) < 0.06).to(torch.int64)
    return wgt, flags


def _types(precision):
    return (torch.complex128, torch.float64) if precision == "fp64" else (torch.complex64,
                                                                         torch.float32)


# ----------------------------------------------------------------------
# what a program holds before the call

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    uvw, freq, centre, cfg = _observation(case, seed)
    if kind == "ng":
        return _prepare_ng(case, seed, uvw, freq, centre, cfg)
    if kind == "weights":
        return _prepare_weights(case, seed, uvw, freq, centre, cfg)
    f = torch.from_numpy(freq).to(DEVICE)
    if kind == "dft":
        lmn, flux = _components(case, seed, freq, cfg)
        return dict(kind=kind, uvw=torch.from_numpy(uvw.reshape(-1, 3)).to(DEVICE), freq=f,
                    lmn=lmn, flux=flux, precision=case["precision"], exact=case["exact"])
    from rascil_gb300 import wgridder
    u = _device_uvw(uvw)
    npix, cell, npol = case["npixel"], cfg["cellsize"], case["npol"]
    cdt, rdt = _types(case["precision"])
    shape = (u.shape[0], f.shape[0], npol)
    half = 0.5 * npix * cell
    s = dict(kind=kind, uvw=u, freq=f, npix=npix, cell=cell, npol=npol, eps=case["epsilon"],
             wstack=case["wstack"], precision=case["precision"])
    s["to_image"] = LINEAR_TO_IQUV if npol == 4 else None
    s["to_vis"] = IQUV_TO_LINEAR if npol == 4 else None
    order = "xy" if kind == "oneshot" else "yx"
    if kind in ("oneshot", "invert", "step", "gains"):
        s["vis"] = _noisy_vis(u, f, npol, half, seed, cdt)
    if kind in ("invert", "step"):
        s["wgt"], s["flags"] = _weights_and_flags(shape, seed, rdt)
    if kind == "oneshot":
        s["vis"] = s["vis"][:, :, 0].contiguous()
        s["wgt"] = _weights_and_flags(shape[:2], seed, rdt)[0]
    if kind in ("oneshot", "predict", "step", "gains"):
        s["model"] = _model(npix, cell, npol, seed, rdt, order)
    if kind == "gains":
        from rascil_gb300.autograd import baseline_antennas
        s["ant1"], s["ant2"] = baseline_antennas(case["nants"], case["ntimes"], DEVICE)
        g = _generator(seed + 2)
        s["model"] = s["model"].requires_grad_(True)
        s["gains"] = torch.view_as_complex(
            torch.randn((case["nants"], case["nchan"], 2), generator=g, device=DEVICE) * 0.05
            + torch.tensor([1.0, 0.0], device=DEVICE)).requires_grad_(True)
    if kind in ("invert", "predict", "gains"):
        s["plan"] = wgridder.Plan(u, f, npix, npix, cell, cell, case["epsilon"], case["wstack"],
                                  npol=npol, precision=case["precision"])
    return s


def _prepare_ng(case, seed, uvw, freq, centre, cfg):
    from rascil_gb300.data_models import create_image
    from rascil_gb300.polarisation import PolarisationFrame
    from rascil_gb300.simulation import make_blockvisibility
    bvis = make_blockvisibility(uvw, freq, centre, cfg)
    g = numpy.random.default_rng(int(seed) + 5)
    bvis["imaging_weight"].data[...] = 0.5 + g.random(bvis.vis.shape)
    bvis["flags"].data[...] = g.random(bvis.vis.shape) < 0.06
    model = create_image(case["npixel"], cfg["cellsize"], centre, frequency=[freq.mean()],
                         polarisation_frame=PolarisationFrame("stokesI"))
    model["pixels"].data[0] = _model(case["npixel"], cfg["cellsize"], 1, seed, torch.float64,
                                     "yx").cpu().numpy()
    return dict(kind="ng", bvis=bvis, model=model)


def _prepare_weights(case, seed, uvw, freq, centre, cfg):
    from rascil_gb300.data_models import BlockVisibility, create_image
    from rascil_gb300.polarisation import PolarisationFrame
    npol = case["npol"]
    frame = PolarisationFrame({1: "stokesI", 2: "linearnp", 4: "linear"}[npol])
    shape = uvw.shape[:2] + (len(freq), npol)
    g = numpy.random.default_rng(int(seed) + 5)
    weight = 0.5 + g.random(shape)
    flags = (g.random(shape) < 0.06).astype(numpy.int64)
    bvis = BlockVisibility(numpy.zeros(shape, dtype=numpy.complex64), uvw, freq, centre, frame,
                           flags=flags, weight=weight, imaging_weight=weight.copy())
    image = create_image(case["npixel"], cfg["cellsize"], centre, frequency=[freq.mean()],
                         channel_bandwidth=[2e8], polarisation_frame=frame)
    return dict(kind="weights", bvis=bvis, image=image, weight=weight.copy(),
                weighting=case["weighting"])


def _snapshots(case):
    from rascil_gb300.simulation import snapshot_batch
    return snapshot_batch(case["nsnap"], seed=case["shapes"], max_vis=case["maxvis"])


def _prepare_batch(case, seed):
    from rascil_gb300.batch import SnapshotBatch
    cdt, rdt = _types(case["precision"])
    snaps, vis, models = [], [], []
    for i, sn in enumerate(_snapshots(case)):
        u = _device_uvw(sn["uvw"])
        f = torch.from_numpy(sn["freq"]).to(DEVICE)
        snaps.append(dict(uvw=u, freq=f, npix=sn["npix"], cell=sn["cell"]))
        vis.append(_noisy_vis(u, f, 1, 0.5 * sn["npix"] * sn["cell"], seed + 31 * i, cdt))
        models.append(_model(sn["npix"], sn["cell"], 1, seed + 31 * i, rdt, "yx"))
    return dict(kind="batch", vis=vis, models=models,
                batch=SnapshotBatch(snaps, case["epsilon"], precision=case["precision"]))


def _components(case, seed, freq, cfg):
    """Direction cosines [k, 3] (l, m, n - 1) and spectra [k, chan, pol]."""
    rng = numpy.random.default_rng(int(seed) + 41)
    k, npol = case["ncomp"], case["npol"]
    lm = rng.uniform(-0.07, 0.07, (k, 2))
    lmn = numpy.concatenate([lm, numpy.sqrt(1 - (lm ** 2).sum(1, keepdims=True)) - 1], axis=1)
    flux = rng.uniform(0.1, 5.0, (k, 1, 1)) * (freq / freq[0])[None, :, None] ** -0.7
    flux = flux * (1.0 + 0.05 * rng.normal(size=(k, 1, npol)) + 0.05j * rng.normal(
        size=(k, 1, npol)))
    return torch.from_numpy(lmn).to(DEVICE), torch.from_numpy(flux).to(DEVICE)


# ----------------------------------------------------------------------
# one pass

def run(s):
    kind = s["kind"]
    if kind == "oneshot":
        from rascil_gb300 import wgridder
        dirty = wgridder.ms2dirty(s["uvw"], s["freq"], s["vis"], s["wgt"], s["npix"], s["npix"],
                                  s["cell"], s["cell"], epsilon=s["eps"],
                                  do_wstacking=s["wstack"])
        vis = wgridder.dirty2ms(s["uvw"], s["freq"], s["model"][0], None, s["cell"], s["cell"],
                                epsilon=s["eps"], do_wstacking=s["wstack"])
        return dict(dirty=dirty, vis=vis)
    if kind == "ng":
        from rascil_gb300.imaging.ng import invert_ng, predict_ng
        predicted = predict_ng(s["bvis"], s["model"])
        image, sumwt = invert_ng(predicted, s["model"])
        return dict(vis=predicted["vis"].data, image=image["pixels"].data, sumwt=sumwt)
    if kind == "invert":
        dirty, sumwt = s["plan"].ms2dirty(s["vis"], wgt=s["wgt"], flags=s["flags"],
                                          polmat=s["to_image"], layout="yx", sumwt=True)
        return dict(dirty=dirty, sumwt=sumwt)
    if kind == "predict":
        return dict(vis=s["plan"].dirty2ms(s["model"], polmat=s["to_vis"], npol_vis=s["npol"],
                                           layout="yx"))
    if kind == "step":
        from rascil_gb300 import wgridder
        with wgridder.Plan(s["uvw"], s["freq"], s["npix"], s["npix"], s["cell"], s["cell"],
                           s["eps"], s["wstack"], npol=s["npol"],
                           precision=s["precision"]) as plan:
            dirty, sumwt = plan.ms2dirty(s["vis"], wgt=s["wgt"], flags=s["flags"],
                                         polmat=s["to_image"], layout="yx", sumwt=True)
            vis = plan.dirty2ms(s["model"], polmat=s["to_vis"], npol_vis=s["npol"], layout="yx")
        return dict(dirty=dirty, sumwt=sumwt, vis=vis)
    if kind == "gains":
        from rascil_gb300.autograd import apply_gains, predict
        vis = apply_gains(predict(s["model"], s["plan"]), s["gains"], s["ant1"], s["ant2"])
        loss = (vis - s["vis"]).abs().pow(2).sum()
        sky_grad, gain_grad = torch.autograd.grad(loss, (s["model"], s["gains"]))
        return dict(loss=loss.detach(), vis=vis.detach(), sky_grad=sky_grad, gain_grad=gain_grad)
    if kind == "batch":
        s["batch"].run_native(s["vis"], s["models"])
        return dict(dirty=list(s["batch"].dirty), pred=list(s["batch"].pred))
    if kind == "dft":
        from rascil_gb300.dft import dft_components
        return dict(vis=dft_components(s["uvw"], s["freq"], s["lmn"], s["flux"],
                                       precision=s["precision"], exact=s["exact"]))
    if kind == "weights":
        from rascil_gb300.imaging.weighting import weight_visibility
        numpy.copyto(s["bvis"]["imaging_weight"].data, s["weight"])  # weights are replaced in place
        weight_visibility(s["bvis"], s["image"], weighting=s["weighting"])
        return dict(imaging_weight=s["bvis"]["imaging_weight"].data)
    raise ValueError(kind)


# ----------------------------------------------------------------------
# what a pass cannot do without

def _gridding_flops(items, npol, epsilon, wstack, planes, npixel):
    """One direction: a support of W cells per dimension, eight floating-point
    operations per cell and polarisation (two complex parts, multiply-add, in
    two dimensions' weights), and a transform of each plane of twice the
    image's side."""
    w = math.ceil(math.log10(1.0 / epsilon)) + 2
    side = 2.0 * npixel
    spread = 4.0 * items * npol * w * w * (w if wstack else 1)
    return spread + planes * npol * 10.0 * side * side * math.log2(side)


def _planes(case, cfg, cell):
    if not case["wstack"]:
        return 1
    r2 = 0.5 * (case["npixel"] * cell) ** 2
    reach = max(spec[-1] for spec in cfg["layout"])
    return 8 + 0.5 * reach * cfg["freq"][1] / C_LIGHT * r2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        size = flops = 0.0
        for sn in _snapshots(case):
            pix = sn["npix"] ** 2
            wmax = numpy.abs(sn["uvw"][..., 2]).max() * sn["freq"].max() / C_LIGHT
            planes = 8 + wmax * 0.5 * (sn["npix"] * sn["cell"]) ** 2
            size += 16.0 * sn["nvis"] + 8.0 * pix + 24.0 * sn["uvw"][..., 0].size
            flops += 2 * _gridding_flops(sn["nvis"], 1, case["epsilon"], True, planes, sn["npix"])
        return {"bytes": float(size), "flops": float(flops)}
    rows = case["nants"] * (case["nants"] - 1) // 2 * case["ntimes"]
    items, npol = rows * case["nchan"], case["npol"]
    from rascil_gb300.simulation import CONFIGS
    cfg = CONFIGS[case["config"]]
    if kind == "dft":
        out = 16.0 if case["precision"] == "fp64" else 8.0
        comp = case["ncomp"]
        # per component and item a complex rotation and a complex multiply-add
        # per polarisation
        return {"bytes": 24.0 * rows + out * items * npol
                + comp * (24.0 + 16.0 * case["nchan"] * npol),
                "flops": comp * items * (6.0 + 8.0 * npol)}
    pix = float(case["npixel"]) ** 2
    if kind == "weights":
        # weight, imaging weight and flag in, imaging weight out (host data)
        return {"bytes": 32.0 * items * npol + 24.0 * rows, "flops": 6.0 * items * npol}
    wide = 2 if case["precision"] == "fp64" else 1
    vis, img = 8.0 * wide * items * npol, 4.0 * wide * pix * npol
    extra = (8.0 + 4.0 * wide) * items * npol  # flags and weights
    one = _gridding_flops(items, npol, case["epsilon"], case["wstack"],
                          _planes(case, cfg, cfg["cellsize"]), case["npixel"])
    size = {"oneshot": 48.0 * rows + 2 * vis + 4.0 * wide * items + 2 * img,
            "ng": 24.0 * rows + 2 * vis + 2 * extra + 2 * img,
            "invert": vis + extra + img, "predict": vis + img,
            "step": 24.0 * rows + 2 * vis + extra + 2 * img,
            "gains": 4 * vis + 2 * img}[kind]
    return {"bytes": size, "flops": one * (1 if kind in ("invert", "predict") else 2)}


# ----------------------------------------------------------------------
# the same in 64 bits, by direct sums

MOST_TERMS = 4.5e10  # sines of a direct sum that stay within some seconds


def _lambdas(uvw, freq):
    """[3, items]: uvw in wavelengths, rows outermost."""
    k = (freq / C_LIGHT)[None, :]
    return torch.stack([(uvw[:, i:i + 1] * k).reshape(-1) for i in range(3)])


def _waves(directions, lam):
    """exp(2 pi i directions . lam), [pixels, items]."""
    turns = directions @ lam
    turns -= torch.round(turns)
    return torch.polar(torch.ones_like(turns), turns.mul_(2.0 * math.pi))


def _dirty_sums(uvw, freq, values, npix, cell, wstack):
    """[npol, y, x] from weighted values [rows, chans, npol] (complex128)."""
    lam = _lambdas(uvw, freq)
    v = values.reshape(-1, values.shape[-1])
    c = (torch.arange(npix, dtype=torch.float64, device=DEVICE) - npix // 2) * cell
    npol, items = v.shape[1], v.shape[0]
    if not wstack:
        out = torch.zeros((npol, npix, npix), dtype=torch.float64, device=DEVICE)
        for a in range(0, items, 65536):
            ex = _waves(c[:, None], lam[:1, a:a + 65536])
            ey = _waves(c[:, None], lam[1:2, a:a + 65536])
            for p in range(npol):
                out[p] += ((ey * v[a:a + 65536, p]) @ ex.T).real
        return out
    y, x = torch.meshgrid(c, c, indexing="ij")
    x, y = x.reshape(-1), y.reshape(-1)
    r2 = x * x + y * y
    nm1 = -r2 / (1.0 + torch.sqrt(1.0 - r2))
    directions = torch.stack([x, y, -nm1], dim=1)
    out = torch.empty((npol, npix * npix), dtype=torch.float64, device=DEVICE)
    step = max(64, int(2.5e8 // items))
    for a in range(0, npix * npix, step):
        out[:, a:a + step] = (_waves(directions[a:a + step], lam) @ v).real.T
    return (out / (1.0 + nm1)).reshape(npol, npix, npix)


def _predict_sums(uvw, freq, sky, npix, cell, wstack):
    """[rows, chans, npol] complex128 of components at pixel centres."""
    x, y, flux = sky
    l = torch.from_numpy((x - npix // 2) * cell).to(DEVICE)
    m = torch.from_numpy((y - npix // 2) * cell).to(DEVICE)
    f = torch.from_numpy(flux).to(DEVICE)
    r2 = l * l + m * m
    nm1 = -r2 / (1.0 + torch.sqrt(1.0 - r2)) if wstack else torch.zeros_like(l)
    directions = torch.stack([l, m, -nm1], dim=1)
    f = (f / (1.0 + nm1)[:, None]).to(torch.complex128)
    lam = _lambdas(uvw, freq)
    out = torch.empty((lam.shape[1], f.shape[1]), dtype=torch.complex128, device=DEVICE)
    for a in range(0, lam.shape[1], 1 << 20):
        out[a:a + (1 << 20)] = _waves(directions, lam[:, a:a + (1 << 20)]).conj().T @ f
    return out.reshape(uvw.shape[0], freq.shape[0], -1)


def _mix(values, matrix):
    if matrix is None:
        return values
    return values @ torch.from_numpy(matrix.T.copy()).to(values.device)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    uvw, freq, centre, cfg = _observation(case, seed)
    f = torch.from_numpy(freq).to(DEVICE)
    if kind == "weights":
        return _exact_weights(case, seed, uvw, freq, cfg)
    if kind == "dft":
        u = torch.from_numpy(uvw.reshape(-1, 3)).to(DEVICE)
        lmn, flux = _components(case, seed, freq, cfg)
        out = torch.empty((u.shape[0], len(freq), case["npol"]), dtype=torch.complex128,
                          device=DEVICE)
        for c in range(len(freq)):
            out[:, c] = _waves(-lmn, u.T * (freq[c] / C_LIGHT)).T @ flux[:, c].to(
                torch.complex128)
        return dict(vis=out)
    u = _device_uvw(uvw)
    npix, cell, npol, wstack = case["npixel"], cfg["cellsize"], case["npol"], case["wstack"]
    items = u.shape[0] * f.shape[0]
    cdt, rdt = _types(case["precision"])
    sky = _sky(npix, cell, npol, seed)
    if rdt == torch.float32:  # the model that the call gets is rounded
        img = _model(npix, cell, npol, seed, rdt, "yx")
        x, y = [torch.from_numpy(a).to(DEVICE) for a in sky[:2]]
        at = torch.unique(y * npix + x)
        sky = ((at % npix).cpu().numpy(), (at // npix).cpu().numpy(),
               img.reshape(npol, -1)[:, at].T.double().cpu().numpy())
    affordable = items * float(npix) ** 2 <= MOST_TERMS or (
        not wstack and items * npol * float(npix) ** 2 <= 1.5e12)
    if kind == "ng":
        g = numpy.random.default_rng(int(seed) + 5)
        weight = 0.5 + g.random(uvw.shape[:2] + (len(freq), 1))
        weight = torch.from_numpy(weight * (g.random(weight.shape) >= 0.06)).to(DEVICE)
        vis = _predict_sums(u, f, sky, npix, cell, wstack)
        image = None
        if affordable:
            w = weight.reshape(u.shape[0], len(freq), 1)
            image = (_dirty_sums(u, f, vis * w, npix, cell, wstack) / w.sum())[None].cpu().numpy()
        return dict(vis=vis.reshape(uvw.shape[:2] + (len(freq), 1)).cpu().numpy(), image=image,
                    sumwt=weight.sum().reshape(1, 1).cpu().numpy())
    got = {}
    if kind in ("oneshot", "predict", "step"):
        vis = _mix(_predict_sums(u, f, sky, npix, cell, wstack),
                   IQUV_TO_LINEAR if npol == 4 else None)
        got["vis"] = vis[:, :, 0] if kind == "oneshot" else vis
    if kind in ("oneshot", "invert", "step"):
        data = _noisy_vis(u, f, npol, 0.5 * npix * cell, seed, cdt)
        got["dirty"] = None
        if kind == "oneshot":
            wgt = _weights_and_flags(data.shape[:2], seed, rdt)[0].double()[:, :, None]
        else:
            wgt, flags = _weights_and_flags(data.shape, seed, rdt)
            wgt = wgt.double() * (1 - flags)
            got["sumwt"] = wgt.sum((0, 1))
        if affordable:
            data = data.to(torch.complex128)
            if kind != "oneshot":
                data = _mix(data * (1 - flags), LINEAR_TO_IQUV if npol == 4 else None)
            dirty = _dirty_sums(u, f, data * wgt, npix, cell, wstack)
            got["dirty"] = dirty[0].T.contiguous() if kind == "oneshot" else dirty
    if kind == "gains":
        a1, a2, gains = _gains_inputs(case, seed)
        vis = _predict_sums(u, f, sky, npix, cell, wstack)
        vis = vis * (gains[a1] * gains[a2].conj())[:, :, None]
        data = _noisy_vis(u, f, npol, 0.5 * npix * cell, seed, cdt).to(torch.complex128)
        got = dict(loss=(vis - data).abs().pow(2).sum(), vis=vis, sky_grad=None, gain_grad=None)
    return got


def _gains_inputs(case, seed):
    a1, a2 = numpy.triu_indices(case["nants"], k=1)
    g = _generator(seed + 2)
    gains = torch.view_as_complex(
        torch.randn((case["nants"], case["nchan"], 2), generator=g, device=DEVICE) * 0.05
        + torch.tensor([1.0, 0.0], device=DEVICE))
    return (torch.from_numpy(numpy.tile(a1, case["ntimes"])).to(DEVICE),
            torch.from_numpy(numpy.tile(a2, case["ntimes"])).to(DEVICE),
            gains.to(torch.complex128))


def _exact_weights(case, seed, uvw, freq, cfg):
    npol, npix, cell = case["npol"], case["npixel"], cfg["cellsize"]
    shape = uvw.shape[:2] + (len(freq), npol)
    g = numpy.random.default_rng(int(seed) + 5)
    weight = 0.5 + g.random(shape)
    flags = (g.random(shape) < 0.06).astype(numpy.int64)
    if case["weighting"] == "natural":
        return dict(imaging_weight=weight)
    deg = numpy.degrees(cell)
    lam = uvw[:, :, None, :] * (freq / C_LIGHT)[None, None, :, None]
    step_u, step_v = [1.0 / (npix * d * numpy.pi / 180.0) for d in (-deg, deg)]
    pu = numpy.rint((lam[..., 0] / step_u + (npix // 2 + 1)) - 1).astype(numpy.int64)
    pv = numpy.rint((lam[..., 1] / step_v + (npix // 2 + 1)) - 1).astype(numpy.int64)
    w = weight * (1 - flags)
    out = numpy.zeros(shape)
    cell_of = (pv * npix + pu).reshape(-1)
    grids = [numpy.bincount(cell_of, weights=w[..., p].reshape(-1), minlength=npix * npix)
             for p in range(npol)]
    f2 = (5.0 * 10.0 ** 0.0) ** 2 * sum(g.sum() for g in grids) / sum((g * g).sum()
                                                                      for g in grids)
    for p in range(npol):
        total = grids[p][cell_of].reshape(shape[:3])
        x = w[..., p]
        with numpy.errstate(divide="ignore", invalid="ignore"):
            y = x * x / total if case["weighting"] == "uniform" else (
                x * (1.0 + f2 * x) / (1.0 + f2 * total))
        out[..., p] = numpy.where(total > 0.0, y, 0.0)
    return dict(imaging_weight=out)
