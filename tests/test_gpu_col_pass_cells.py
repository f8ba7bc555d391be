"""The column and FP64 row slice passes on cells of unequal sampling, and over
several tiles a block.

Unequal sampling: the band limit is set by the coarser side, so along the other one
more columns (or rows) are removed than the third of a square cell's, some of them
inside a tile.  FP32 against FP64, FP64 against the plain per-step path, the exit
wave outside the aperture and the ADF signal.  A transform of up to 4096 points
rounds to at most 12 x 6e-8 of its result, three slices run four each, 8.6e-6 if
every error added up, twice that for the ADF signal's square; a lost column is an
error of the order of 1.  FP64, likewise: 12 x 12 x 1.1e-16 = 1.6e-14 of the whole
wave, of which the part outside the aperture is above 1e-4.

Several tiles: a batch that takes every block through its buffers often enough
for both parities of each (columns up to 512 points: at least twice the buffers
and one; beyond: three tiles) against one probe a launch, one tile or two a block,
bit for bit."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu

ALPHA = 0.010


def _setup(nx, ny, precision, raster_n, batch=0, side=(1.0, 1.0), depth=6.0):
    box = (nx * 0.1 * side[0], ny * 0.1 * side[1], depth)
    n = max(6, int(0.01 * box[0] * box[1] * box[2]))
    q = np.random.default_rng(8).uniform(0.0, 1.0, (n, 3)) * box
    grid = msf.Grid(nx=nx, ny=ny, voltage=200000.0, xperiod=box[0], yperiod=box[1],
                    zperiod=depth, dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0,
                    ymin=0.0, zmin=0.0, min_slice=2.0)
    xp = np.arange(raster_n[0]) * (box[0] / raster_n[0])
    yp = np.arange(raster_n[1]) * (box[1] / raster_n[1])
    raster = msf.Raster(len(xp), len(yp), xp.ctypes.data_as(msf._dp), yp.ctypes.data_as(msf._dp))
    raster.keep = (xp, yp)
    ctx = msf.Context(precision=precision, batch=batch)
    spec = ctx.specimen(grid, q, np.full(n, 14, np.uint32))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=ALPHA)
    det = msf.Detect(outputs=msf.OUT_ADF_IMAGE, det_inner=0.04, det_outer=0.2, dr=1.0)
    return ctx, spec, optics, raster, det, box


def _wave(nx, ny, precision, side, plain=False):
    ctx, spec, optics, raster, det, box = _setup(nx, ny, precision, (2, 1), side=side)
    res = (ctx.run_plain if plain else ctx.run)(spec, optics, raster, det, want_final_psi=True)
    lam = msf.wavelength(200000.0)[0]
    kx, ky = (np.fft.fftfreq(n, b / n) for n, b in ((nx, box[0]), (ny, box[1])))
    k2 = kx[:, None] ** 2 + ky[None, :] ** 2
    bw = (2.0 / 3.0) * min(nx / (2 * box[0]), ny / (2 * box[1]))
    psi = res.final_psi_2d[..., 0] + 1j * res.final_psi_2d[..., 1]
    assert not psi[k2 >= bw * bw].any()
    return psi[(k2 < bw * bw) & (k2 * lam * lam > (1.01 * ALPHA) ** 2)], res.adf_image


GRIDS = [(64, 64), (128, 256), (256, 128), (512, 64), (1024, 128), (2048, 64), (4096, 64),
         (64, 4096)]


@pytest.mark.parametrize("side", [(1.0, 0.7), (0.7, 1.0), (1.0, 0.93)])
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_fp32_on_unequal_sampling(nx, ny, side):
    (got, adf), (want, adf64) = _wave(nx, ny, "fp32", side), _wave(nx, ny, "fp64", side)
    assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(want)
    np.testing.assert_allclose(adf, adf64, rtol=2e-5)


@pytest.mark.parametrize("side", [(1.0, 0.7), (0.7, 1.0), (1.0, 0.93)])
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_fp64_on_unequal_sampling(nx, ny, side):
    (got, adf), (want, plain) = _wave(nx, ny, "fp64", side), _wave(nx, ny, "fp64", side, True)
    assert np.linalg.norm(got - want) < 1e-9 * np.linalg.norm(want)
    np.testing.assert_allclose(adf, plain, rtol=1e-9)


# about 2/3 of ny is live; FP32 tiles hold 16 columns up to 1024 points, then 8 and
# 4, FP64 ones half as many; 592, 592, 296 and 148 blocks from 64 to 512 points in
# FP32, 592, 296, 148 and 148 in FP64, 148 beyond
@pytest.mark.parametrize("precision,nx,ny,probes", [
    ("fp32", 64, 4096, (8, 4)), ("fp32", 128, 4096, (8, 4)), ("fp32", 256, 2048, (8, 4)),
    ("fp32", 512, 1024, (8, 4)), ("fp32", 1024, 256, (8, 8)), ("fp32", 2048, 128, (8, 8)),
    ("fp32", 4096, 64, (8, 8)), ("fp64", 64, 2048, (8, 4)), ("fp64", 128, 1024, (8, 8)),
    ("fp64", 256, 512, (8, 8)), ("fp64", 512, 512, (8, 4)), ("fp64", 1024, 128, (8, 8)),
    ("fp64", 2048, 64, (8, 8)), ("fp64", 4096, 64, (8, 4))])
def test_many_tiles_a_block_equal_one(precision, nx, ny, probes):
    n = probes[0] * probes[1]
    sums = []
    for batch in (n, 1):
        ctx, spec, optics, raster, det, _ = _setup(nx, ny, precision, probes, batch, depth=4.0)
        sums.append(ctx.run_partial(spec, optics, raster, det, 0, n))
    for key in ("amp", "inten"):
        np.testing.assert_array_equal(sums[0][key], sums[1][key], err_msg=key)
        assert (sums[0][key] > 0).all()
