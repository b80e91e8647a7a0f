"""O(N^2) FP64 potential energy (src/c/diagnostics/numerics.c:83-116) at the
edges of the kernel's rectangles, against the oracle's scalar sum.  Every term
has the same sign, so the sums differ by rounding alone: at most ~1e3 roundings
of 1.1e-16 along the device's longest chain, and on the oracle's sequential sum
of 4e7 terms a random walk of 7e-13."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def to_system(nb, p):
    return nb.ParticleSystem(*[getattr(p, f).copy() for f in O.FIELDS])


@pytest.mark.parametrize("n", [1, 2, 3, 127, 128, 129, 255, 1025, 8191, 8192, 8193, 8449])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_potential_energy_at_rectangle_edges(cuda, ctx, n, eps):
    p = O.preset_parallel("globular_cluster", max(n, 2), 5)
    p = O.Particles(*[getattr(p, f)[:n].copy() for f in O.FIELDS])
    ctx.upload(to_system(cuda, p))
    _, pe = ctx.diagnostics(cuda.gravity_init(1.0, eps), potential=True)
    ref = O.potential_energy(p, 1.0, eps)
    assert abs(pe - ref) <= 2e-12 * abs(ref)


@pytest.mark.parametrize("scale", [1e-155, 1e-150, 1e150])
def test_potential_energy_at_extreme_distances(cuda, ctx, scale):
    """Squared distances that underflow, are subnormal or nearly overflow take
    the library reciprocal root."""
    p = O.preset_parallel("globular_cluster", 300, 5)
    for f in ("x", "y", "z"):
        getattr(p, f)[:] *= scale
    ctx.upload(to_system(cuda, p))
    _, pe = ctx.diagnostics(cuda.gravity_init(1.0, 0.0), potential=True)
    ref = O.potential_energy(p, 1.0, 0.0)
    # at 1e-155 the squared distances (down to 1e-313) are subnormal, spaced 5e-324
    assert abs(pe - ref) <= (1e-10 if scale == 1e-155 else 2e-12) * abs(ref)


def test_potential_energy_of_coincident_particles_is_infinite(cuda, ctx):
    p = O.preset_parallel("globular_cluster", 400, 5)
    for f in ("x", "y", "z"):
        getattr(p, f)[391] = getattr(p, f)[7]
    ctx.upload(to_system(cuda, p))
    _, pe = ctx.diagnostics(cuda.gravity_init(1.0, 0.0), potential=True)
    assert pe == -np.inf
