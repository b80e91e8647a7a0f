"""The relative opening test of a plugin call whose accelerations come in while the
tree is built: the same forces and counts, bit for bit, as a resident evaluation
that reads them before the sort, with pageable and page-locked arrays, at both
forms of the sort, and for accelerations that are all zero or not finite."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def page_locked(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("kind", ["forces", "zero", "nan"])
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [16384, 16385, 20480, 20481, 98304, 98305, 300001])
def test_plugin_call_equals_resident_evaluation(cuda, ctx, n, pinned, kind):
    p = O.preset_parallel("galaxy_collision", n, 13)
    s = cuda.ParticleSystem.zeros(n, page_locked if pinned else None)
    for f in O.FIELDS:
        getattr(s, f)[:] = getattr(p, f)
    g = cuda.gravity_init(1.0, 0.02)
    if kind == "forces":
        ctx.upload(s)
        ctx.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
        s.ax[:], s.ay[:], s.az[:] = ctx.download_accelerations().T
    else:
        rng = np.random.default_rng(n)
        for a in (s.ax, s.ay, s.az):
            a[:] = 0.0 if kind == "zero" else rng.normal(size=n)
        if kind == "nan":
            s.ay[n // 3], s.az[n // 2] = np.nan, np.inf
    ctx.theta = 1.0
    ctx.set_relative_opening(0.003)
    old = s.acc().copy()
    ctx.upload(s)
    ctx.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
    want, stats = ctx.download_accelerations(), ctx.stats()
    for _ in range(2):
        s.ax[:], s.ay[:], s.az[:] = old.T
        got = cuda.n_body_sim_pro_barnes_hut_compute_acceleration_cuda(s, g, ctx)
        np.testing.assert_array_equal(got, want)
        now = ctx.stats()
        assert all(now[k] == stats[k] for k in stats if not k.endswith("seconds"))
