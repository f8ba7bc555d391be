"""The launch count a call reports includes the ring means of its finish where
that kernel runs, and only there."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_ring_means_are_counted_where_they_launch(precision):
    n, box = 64, 6.4
    q = np.random.default_rng(7).uniform(0.0, 1.0, (20, 3)) * (box, box, 4.0)
    grid = msf.Grid(nx=n, ny=n, voltage=200000.0, xperiod=box, yperiod=box, zperiod=4.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    xp = np.array([0.0, 2.0, 4.0])
    raster = msf.Raster(3, 1, xp.ctypes.data_as(msf._dp), xp.ctypes.data_as(msf._dp))
    optics = msf.Optics(corrected=0, cs3=1.3e7, cs5=0.0, defocus=400.0, alpha_max=0.010)
    ring, pixel = (msf.Detect(outputs=msf.OUT_ADF_IMAGE | mode, det_inner=0.04, det_outer=0.2,
                              dr=1.0) for mode in (msf.OUT_V_OMEGA, msf.OUT_V_RE))
    ctx = msf.Context(precision=precision)
    spec = ctx.specimen(grid, q, np.full(len(q), 14, np.uint32))

    def extra(call):
        """Launches the pixel mode adds to the same call's ring mode."""
        return call(pixel) - call(ring)

    # one batch: the pixel sums are one launch, the ring means of the finish another
    assert extra(lambda d: ctx.run(spec, optics, raster, d).kernel_launches) == 2
    assert extra(lambda d: ctx.run_md([spec], 1, optics, raster, d).kernel_launches) == 2
    # sums alone, finished elsewhere
    assert extra(lambda d: ctx.run_partial(spec, optics, raster, d, 0, 3)["kernel_launches"]) == 1
    if precision == "fp32":  # a lane's detection is three launches in either mode
        job = lambda d: ctx.run_batch([(spec, optics, raster, d)])[0].kernel_launches
        assert extra(job) == 1
    else:
        plain = lambda d: ctx.run_plain(spec, optics, raster, d).kernel_launches
        assert extra(plain) == 3 + 1  # one launch a probe, and the means
