"""Phase timings from the GPU's clock, and the counts of an advance's last step,
at both forms of the sort: the phases fit into the total, which two events
measure (to a few ticks of the clock, 0.01 ms), and an advance of several steps reports the evaluation at its final positions."""
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
PHASES = ("bounds_ms", "keys_ms", "sort_ms", "build_ms", "moments_ms", "walk_ms", "integrate_ms")
COUNTS = ("node_count", "leaf_count", "internal_node_count", "accepted_approximations",
          "exact_interactions", "maximum_depth")


@pytest.mark.parametrize("n", [2, 2000, 98304, 98305])
def test_phases_and_counts_of_the_last_evaluation(cuda, ctx, n):
    p = O.preset_parallel("globular_cluster", n, 5)
    g = cuda.gravity_init(1.0, 0.05)
    ctx.upload(cuda.ParticleSystem(*[getattr(p, f).copy() for f in O.FIELDS]))
    ctx.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
    ctx.advance(g, 1e-2, 3, cuda.Algorithm.BARNES_HUT)
    for _ in range(2):  # the advance's last evaluation, then one at the same positions
        t = ctx.timings()
        assert all(t[k] >= 0.0 for k in PHASES)
        assert 0.0 < sum(t[k] for k in PHASES) <= t["total_ms"] + 0.01
        s = ctx.stats()
        counts = [s[k] for k in COUNTS]
        assert counts[0] >= counts[1] > 0
        ctx.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
    assert [ctx.stats()[k] for k in COUNTS] == counts
