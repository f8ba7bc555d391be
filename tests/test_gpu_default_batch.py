"""Probes per launch when neither the caller nor the tuner chose them, in a
context whose memory is bounded.  The default of 256 probes at 512^2 takes 0.5
GiB of FP32 wavefields; a bound that holds 64 is enough for the same raster.  A
probe's sums do not depend on the batch it runs in, so the results equal an
unbounded context's bit for bit."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu

MIB = 1 << 20
OUTPUTS = msf.OUT_ADF_IMAGE | msf.OUT_V_OMEGA | msf.OUT_V_RE
MTF = np.array([1.0, 0.6, 0.2])
MTF_DOMAIN_SQR = np.array([0.0, 5.0, 10.0]) ** 2


def _run(precision, kind, **options):
    n, box = 512, 51.2
    q = np.random.default_rng(5).uniform(0.0, 1.0, (60, 3)) * (box, box, 4.0)
    grid = msf.Grid(nx=n, ny=n, voltage=200000.0, xperiod=box, yperiod=box, zperiod=4.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    ctx = msf.Context(precision=precision, **options)
    spec = ctx.specimen(grid, q, np.full(len(q), 14, np.uint32))
    xp = np.arange(16) * (box / 16)
    raster = msf.Raster(16, 16, xp.ctypes.data_as(msf._dp), xp.ctypes.data_as(msf._dp))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010)
    det = msf.Detect(outputs=OUTPUTS, det_inner=0.04, det_outer=0.2, dr=1.0)
    if kind == "mtf":
        det.n_mtf, det.mtf_resolution = len(MTF), 20.0
        det.mtf, det.mtf_domain_sqr = (a.ctypes.data_as(msf._dp) for a in (MTF, MTF_DOMAIN_SQR))
    if kind == "partial":
        return ctx.run_partial(spec, optics, raster, det, 0, 256)
    if kind == "md":
        res = ctx.run_md([spec], 2, optics, raster, det)
    else:
        res = ctx.run(spec, optics, raster, det, want_final_psi=True)
    return {"adf": res.adf_image, "final": res.final_psi, "first": res.first_psi, **res.v}


def _same(got, want):
    for key in ("adf", "final", "first", "V_omega", "V_re", "amp", "inten", "acc_a", "acc_i"):
        if want.get(key) is not None:
            np.testing.assert_array_equal(got[key], want[key], err_msg=key)


@pytest.mark.parametrize("precision,kind", [("fp32", "run"), ("fp64", "run"),
                                            ("fp32", "partial")])
def test_bound_that_holds_64_probes(precision, kind):
    """The smallest bound (to 1 MiB) under which 64 probes a launch run is
    enough for the default."""
    waves = 64 * 2 * (2 if precision == "fp64" else 1)  # MiB
    low, high = waves, waves + 128
    _run(precision, kind, batch=64, hbm_budget=high * MIB)
    while high - low > 1:
        mid = (low + high) // 2
        try:
            _run(precision, kind, batch=64, hbm_budget=mid * MIB)
            high = mid
        except msf.MsfError:
            low = mid
    _same(_run(precision, kind, hbm_budget=high * MIB), _run(precision, kind))


@pytest.mark.parametrize("kind", ["mtf", "md"])
def test_bound_below_the_batch_of_a_long_plan(kind):
    """FP64 planes beside the wavefields (4 MiB a probe each): 192 MiB hold
    about 25 probes of them."""
    _same(_run("fp32", kind, hbm_budget=192 * MIB), _run("fp32", kind))


def test_second_raster_of_a_bounded_context():
    """A block kept from an earlier raster is no reason for a batch beyond the
    bound."""
    n, box = 256, 25.6
    q = np.random.default_rng(6).uniform(0.0, 1.0, (30, 3)) * (box, box, 4.0)
    grid = msf.Grid(nx=n, ny=n, voltage=200000.0, xperiod=box, yperiod=box, zperiod=4.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    xp = np.arange(16) * (box / 16)
    raster = msf.Raster(16, 16, xp.ctypes.data_as(msf._dp), xp.ctypes.data_as(msf._dp))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010)
    det = msf.Detect(outputs=OUTPUTS, det_inner=0.04, det_outer=0.2, dr=1.0)
    runs = []
    for budget in (0, 80 * MIB):
        ctx = msf.Context(precision="fp32", hbm_budget=budget)
        spec = ctx.specimen(grid, q, np.full(len(q), 14, np.uint32))
        for _ in range(2):
            runs.append(ctx.run(spec, optics, raster, det))
        md = ctx.run_md([spec], 1, optics, raster, det)
        runs.append(md)
    for got, want in zip(runs[3:], runs[:3]):
        np.testing.assert_array_equal(got.adf_image, want.adf_image)
        np.testing.assert_array_equal(got.v["V_re"], want.v["V_re"])
