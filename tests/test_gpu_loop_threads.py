"""On-chip loops from two host threads, each with its own context and a launch that
takes every SM, and beside 3D steps of a third: every run gives the bits it gives
alone (a cooperative launch starts when all its blocks can, so the loops take turns)."""
import threading

import numpy as np
import pytest

import test_gpu_loop2d as loop2d

pytestmark = pytest.mark.gpu


def _run(pkg, s, runs, out, key):
    try:
        ctx = pkg.Context(0)
        plan = ctx.plan(s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"],
                        s["posrecs"])
        for _ in range(runs):
            plan.reset()
            plan.run()
            out.setdefault(key, []).append((plan.traces(), plan.field()))
        plan.close()
        ctx.close()
    except Exception as e:  # reported by the main thread
        out[key] = e


def test_two_loops_and_a_3d_run(pkg):
    jobs = {"loop f32": loop2d._setup(pkg, (1573, 787, 20, True), "f32", 1),
            "loop f64": loop2d._setup(pkg, (1003, 803, 20, False), "f64", 2)}
    n = (120, 110, 100)
    srcs = pkg.Sources([[m * 5.0 for m in n]], [0.02], [pkg.rickersource1D], 30.0)
    jobs["3d"] = pkg.prepare([(m - 1) * 10.0 for m in n], None, np.full(n, 2000.0), srcs,
                             pkg.Receivers([[m * 5.0 + 20.0 for m in n]]), halo=12, ppw=1e-9,
                             precision="f32", nt=200)
    alone, together = {}, {}
    for key, s in jobs.items():
        _run(pkg, s, 1, alone, key)
    threads = [threading.Thread(target=_run, args=(pkg, s, 12, together, key))
               for key, s in jobs.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for key in jobs:
        assert isinstance(alone[key], list), alone[key]
        assert isinstance(together[key], list), together[key]
        for traces, field in together[key]:
            np.testing.assert_array_equal(traces, alone[key][0][0])
            np.testing.assert_array_equal(field, alone[key][0][1])
