"""A specimen may outlive its context (a garbage collector destroys them in
either order): destroying it then touches nothing of the context, and leaves the
thread's CUDA state as it was for the next one."""
import numpy as np
import pytest

import msf

pytestmark = pytest.mark.gpu


def test_specimen_destroyed_after_its_context():
    box = 6.4
    q = np.random.default_rng(1).uniform(0.0, 1.0, (20, 3)) * (box, box, 4.0)
    grid = msf.Grid(nx=64, ny=64, voltage=200000.0, xperiod=box, yperiod=box, zperiod=4.0,
                    dupe_x=1, dupe_y=1, dupe_z=1, replicate_atoms=0, xmin=0.0, ymin=0.0,
                    zmin=0.0, min_slice=2.0)
    for _ in range(4):
        ctx = msf.Context()
        spec = ctx.specimen(grid, q, np.full(len(q), 14, np.uint32))
        ctx.close()
        overwritten = [bytearray(b"\x7f" * n) for n in range(400, 1400, 8)]  # freed memory's reuse
        spec.close()
        del overwritten
