"""Detection steps that run on the device: the annulus pixel list (runs found
by bisection, expanded by a kernel) and the ring sums of the pixel FEM modes.

Both replace host loops bit for bit: the ADF sum of a plan with an annulus cut
anywhere equals numpy's sum of the same exit wave's pixels to FP64 rounding of
the sum (1e-12), and the pixel modes of msf_run equal msf_finish's host sums of
the same per-pixel sums exactly."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu


def _setup(nx, ny, box, precision, outputs, inner, outer):
    q = np.random.default_rng(3).uniform(0.0, 1.0, (40, 3)) * (box[0], box[1], 4.0)
    grid = msf.Grid(nx=nx, ny=ny, voltage=200000.0, xperiod=box[0], yperiod=box[1], zperiod=4.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    ctx = msf.Context(precision=precision)
    spec = ctx.specimen(grid, q, np.full(len(q), 14, np.uint32))
    xp, yp = np.array([0.0, box[0] / 3]), np.array([0.0, box[1] / 2, box[1] * 0.9])
    raster = msf.Raster(2, 3, xp.ctypes.data_as(msf._dp), yp.ctypes.data_as(msf._dp))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010)
    det = msf.Detect(outputs=outputs, det_inner=inner, det_outer=outer, dr=1.0)
    return ctx, spec, optics, raster, det, (xp, yp)


# square, rectangular and anisotropic cells; an annulus inside the band limit,
# one that starts at k = 0 (only the zero pixel outside), an empty one, and one
# that takes every pixel
@pytest.mark.parametrize("nx,ny,box", [(64, 64, (6.4, 6.4)), (128, 64, (12.8, 12.8)),
                                       (64, 256, (6.4, 12.8))])
@pytest.mark.parametrize("inner,outer", [(0.02, 0.1), (0.0, 0.05), (0.05, 0.05), (-1.0, 1e3)])
def test_annulus_sum_matches_exit_wave(nx, ny, box, inner, outer):
    ctx, spec, optics, raster, det, keep = _setup(nx, ny, box, "fp64", msf.OUT_ADF_IMAGE, inner,
                                                  outer)
    res = ctx.run(spec, optics, raster, det, want_final_psi=True)
    lam = msf.wavelength(200000.0)[0]
    kx, ky = (np.fft.fftfreq(n, b / n) for n, b in ((nx, box[0]), (ny, box[1])))
    k2 = kx[:, None] ** 2 + ky[None, :] ** 2
    psi = res.final_psi_2d[..., 0] ** 2 + res.final_psi_2d[..., 1] ** 2
    want = psi[(k2 > inner / lam) & (k2 <= outer / lam)].sum()
    np.testing.assert_allclose(res.adf_image[-1], want, rtol=1e-12)


@pytest.mark.parametrize("nx,ny,box", [(64, 64, (6.4, 6.4)), (256, 64, (25.6, 6.4)),
                                       (512, 512, (51.2, 51.2))])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_pixel_modes_equal_host_finish(nx, ny, box, precision):
    outputs = msf.OUT_ADF_IMAGE | msf.OUT_V_RE | msf.OUT_OMEGA_VIMAGE | msf.OUT_V_GT17 | msf.OUT_V_RBAR
    ctx, spec, optics, raster, det, keep = _setup(nx, ny, box, precision, outputs, 0.04, 0.2)
    got = ctx.run(spec, optics, raster, det, want_means=True)
    part = ctx.run_partial(spec, optics, raster, det, 0, 6)
    want = msf.finish(spec.grid, optics, raster, det, part["amp"], part["inten"], part["acc_a"],
                      part["acc_i"], want_means=True)
    for m, v in want.v.items():
        assert np.array_equal(got.v[m], v, equal_nan=True), m
    assert np.array_equal(got.mean_amplitude, want.mean_amplitude)
    assert np.array_equal(got.mean_intensity, want.mean_intensity)


# The vacuum part of an FP32 exit wave: its phases come from masked integers and
# it is kept inside the aperture only.  Long and short sides both ways, shifts
# up to nearly a side; apertures of one pixel, of some, and past the band limit.
# FP32 rounds the scattered part alone: log2(N) eps = 7e-7 a transform, 4
# transforms a slice, 2 slices, 6e-6 if every error added up.
@pytest.mark.parametrize("nx,ny", [(64, 64), (64, 4096), (4096, 64), (256, 128)])
@pytest.mark.parametrize("alpha", [1e-5, 0.010, 1.0])
def test_fp32_exit_wave_matches_fp64(nx, ny, alpha):
    waves = []
    for precision in ("fp32", "fp64"):
        ctx, spec, optics, raster, det, keep = _setup(nx, ny, (nx * 0.1, ny * 0.1), precision,
                                                      msf.OUT_ADF_IMAGE, 0.04, 0.2)
        optics.alpha_max = alpha
        waves.append(ctx.run(spec, optics, raster, det, want_final_psi=True).final_psi_2d)
    err = np.linalg.norm(waves[0] - waves[1]) / np.linalg.norm(waves[1])
    assert err < 1e-5, err


# Ring, annulus and pixel sums gather several pixels or probes at a time: counts
# that are no multiple of them (1, 3, 5, 6 probes; short rings), each against the
# same sums of one probe at a time, which add the same values in the same order
# within a segment (exact) and the probes' planes in raster order (1e-14 of FP64
# rounding for 6 of them).
@pytest.mark.parametrize("nx,ny,box", [(64, 64, (6.4, 6.4)), (256, 128, (25.6, 12.8))])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 3, 5, 6])
def test_sums_of_a_batch_equal_single_probes(nx, ny, box, precision, n):
    outputs = msf.OUT_ADF_IMAGE | msf.OUT_V_RE | msf.OUT_OMEGA_VIMAGE
    ctx, spec, optics, raster, det, keep = _setup(nx, ny, box, precision, outputs, 0.04, 0.2)
    whole = ctx.run_partial(spec, optics, raster, det, 0, n)
    one = [ctx.run_partial(spec, optics, raster, det, k, k + 1) for k in range(n)]
    for key in ("amp", "inten"):
        assert np.array_equal(whole[key], np.concatenate([o[key] for o in one])), key
    for key in ("acc_a", "acc_i"):
        np.testing.assert_allclose(whole[key], sum(o[key] for o in one), rtol=1e-14)
