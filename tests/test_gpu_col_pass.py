"""The column slice pass (kernels_col.cuh) and the FP64 row pass
(kernels_row64.cu) at every length they support: FP32 against the FP64 passes
of the same raster, FP64 against the plain per-step path.

FP32 tolerance: a packed transform of up to 4096 points rounds to at most about
log2(N) eps = 12 x 6e-8 of its result; three slices run four each (two per
axis), 8.6e-6 if every error added up, and the ADF signal is quadratic in the
wave: 2e-5 relative."""
import numpy as np
import pytest

import msf
import specimen

pytestmark = pytest.mark.gpu


def _run(nx, ny, precision, raster_n, batch, plain=False):
    box = (nx * 0.1, ny * 0.1, 6.0)
    n = max(6, int(0.01 * box[0] * box[1] * box[2]))
    q = specimen.amorphous_positions(n, box, seed=5)
    grid = msf.Grid(nx=nx, ny=ny, voltage=200000.0, xperiod=box[0], yperiod=box[1], zperiod=6.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    xp = np.arange(raster_n[0]) * (box[0] / raster_n[0])
    yp = np.arange(raster_n[1]) * (box[1] / raster_n[1])
    ctx = msf.Context(precision=precision, batch=batch)
    spec = ctx.specimen(grid, q, np.full(n, 14, np.uint32))
    run = ctx.run_plain if plain else ctx.run
    return run(spec, msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010),
               msf.Raster(len(xp), len(yp), xp.ctypes.data_as(msf._dp),
                          yp.ctypes.data_as(msf._dp)),
               msf.Detect(outputs=msf.OUT_ADF_IMAGE, det_inner=0.04, det_outer=0.2, dr=1.0))


# nx: each kernel's lengths; ny: the fewest column groups (64), an uneven split
# of them over the grid, and as many as fill every persistent block; probes: one,
# an odd number, and a batch with a remainder
@pytest.mark.parametrize("nx,ny,raster,batch", [
    (64, 64, (1, 1), 0), (64, 512, (3, 5), 4), (128, 64, (3, 3), 0), (256, 64, (1, 1), 0),
    (256, 1024, (5, 5), 8), (512, 64, (3, 1), 0), (512, 512, (3, 3), 4), (1024, 64, (1, 1), 0),
    (1024, 256, (3, 5), 7), (2048, 64, (3, 1), 0), (2048, 256, (3, 3), 4), (4096, 64, (1, 1), 0),
    (4096, 128, (3, 1), 2)])
def test_column_pass_matches_fp64(nx, ny, raster, batch):
    got, want = _run(nx, ny, "fp32", raster, batch), _run(nx, ny, "fp64", raster, batch)
    assert want.adf_image.min() > 0
    np.testing.assert_allclose(got.adf_image, want.adf_image, rtol=2e-5)


# FP64 at every length, where the packed FP32 pass and the FP64 one share their
# kernels: against the plain per-step path (other transforms throughout).  Both
# are FP64: 12 stages x 4 transforms x 3 slices x 1.1e-16, twice for the ADF
# signal's square, times the cancellation of a scattered part 1e-3 of the
# direct beam, stays under 1e-10.
@pytest.mark.parametrize("nx,ny,raster,batch", [
    (64, 64, (1, 1), 0), (64, 4096, (1, 2), 0), (128, 64, (3, 3), 2), (256, 1024, (3, 3), 4),
    (512, 128, (3, 1), 0), (1024, 512, (1, 3), 2), (2048, 256, (1, 1), 0), (4096, 2048, (1, 1), 0)])
def test_fp64_passes_match_plain_path(nx, ny, raster, batch):
    got = _run(nx, ny, "fp64", raster, batch)
    want = _run(nx, ny, "fp64", raster, batch, plain=True)
    np.testing.assert_allclose(got.adf_image, want.adf_image, rtol=1e-10)
