"""The device time that awc_batch_run reports covers the steps: a batch's first run
through the loop, which prepares the loop's tables, reports what later ones do."""
import numpy as np
import pytest

import test_gpu_loop2d as loop2d

pytestmark = pytest.mark.gpu


def test_first_run_reports_its_steps_only(pkg, ctx):
    setups = [loop2d._setup(pkg, (200, 150, 10, True), "f32", seed=k) for k in range(4)]
    p = setups[0]["problem"]
    model = pkg.Problem(ndim=2, precision=p.precision, nx=p.nx, ny=p.ny, nz=1, halo=p.halo,
                        freetop=p.freetop, dx=p.dx, dy=p.dy, dz=1.0, dt=p.dt, nt=p.nt, nsrc=0,
                        nrec=0)
    first, later = [], []
    for _ in range(6):
        batch = pkg.Batch(ctx, [model], [setups[0]["vel"]], setups, [0] * 4)
        assert batch.launch_count(8) == 1
        first.append(batch.run(8))
        batch.reset()
        later.append(batch.run(8))
        batch.close()
    print(first, later)
    # the first batch's run loads the kernel; three times covers the scatter of
    # 20 us (the tables take 0.7 ms, a run 0.03)
    assert np.min(first[1:]) <= 3.0 * np.min(later[1:])
