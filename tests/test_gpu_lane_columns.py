"""Rasters of one grid size whose cells differ slightly in aspect share a slot
lane.  Their band limits keep the same column groups but remove different
columns within them (the first cell's more), so a lane that skipped the first
one's columns for both would drop k-space columns of the second.  Each raster
of the mix gives the bits it gives alone: a probe's arithmetic does not depend
on its companions, and skipping a removed column leaves the zeros that computing
it would."""
import time

import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu


def _job(nx, ny, aspect, seed, raster_n=3):
    """(grid, positions, atomic numbers, optics, raster, detect) of an
    nx x ny grid over a cell whose y side is `aspect` times that of square
    pixels."""
    box = np.array([nx * 0.1, ny * 0.1 * aspect, 6.0])
    rng = np.random.default_rng(seed)
    q = rng.uniform(0.0, 1.0, (max(6, int(0.01 * box.prod())), 3)) * box
    grid = msf.Grid(nx=nx, ny=ny, voltage=200000.0, xperiod=box[0], yperiod=box[1],
                    zperiod=box[2], dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0,
                    ymin=0.0, zmin=0.0, min_slice=2.0)
    xp = np.arange(raster_n) * (box[0] / raster_n)
    yp = np.arange(raster_n) * (box[1] / raster_n)
    raster = msf.Raster(raster_n, raster_n, xp.ctypes.data_as(msf._dp), yp.ctypes.data_as(msf._dp))
    raster.keep = (xp, yp)
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010)
    detect = msf.Detect(outputs=msf.OUT_ADF_IMAGE | msf.OUT_V_OMEGA, det_inner=0.04,
                        det_outer=0.2, dr=1.0)
    return grid, q, np.full(len(q), 14, np.uint32), optics, raster, detect


def _same(got, want):
    np.testing.assert_array_equal(got.adf_image, want.adf_image)
    np.testing.assert_array_equal(got.v["V_omega"], want.v["V_omega"])


# cells whose column groups agree: 16 columns a group up to 1024 points, 8 at
# 2048, 4 at 4096
@pytest.mark.parametrize("nx,ny,aspect", [
    (64, 64, 0.9), (128, 128, 0.9), (256, 256, 0.95), (1024, 1024, 0.99), (2048, 64, 0.9),
    (4096, 128, 0.97), (64, 4096, 0.9975)])
def test_batch_of_two_aspects(nx, ny, aspect):
    ctx = msf.Context(precision="fp32")
    jobs = [_job(nx, ny, aspect, 1), _job(nx, ny, 1.0, 2)]
    runs = [(ctx.specimen(g, q, z), *rest) for g, q, z, *rest in jobs]
    assert runs[0][0].live_columns() < runs[1][0].live_columns()
    alone = [ctx.run_batch([r], slots=4)[0] for r in runs]
    for got, want in zip(ctx.run_batch(runs, slots=4), alone):
        _same(got, want)


@pytest.mark.parametrize("n,aspect", [(64, 0.9), (256, 0.95)])
def test_server_with_two_aspects(n, aspect):
    def serve(jobs):
        server = msf.Server(slots=4)
        tickets = [server.submit(*j) for j in jobs]
        outs = []
        for t in tickets:
            r, end = None, time.time() + 120
            while r is None:
                assert time.time() < end, "request did not finish"
                r = server.poll(t, wait_ms=200)
            outs.append(r)
        server.close()
        return outs

    jobs = [_job(n, n, aspect, 3, raster_n=6), _job(n, n, 1.0, 4, raster_n=6)]
    alone = [serve([j])[0] for j in jobs]
    for got, want in zip(serve(jobs), alone):
        _same(got, want)
