"""Plugin calls of small systems: page-locked and pageable arrays, both
algorithms, at the edges of the two-kernel all-pairs path (clusters of 256
sources, targets of 128, up to 2047 particles) and of the staging rows, against
the resident evaluation of the same state and the FP64 sums.

Both paths sum the same FP32 tiles of 128 sources in the same order and differ
in the grouping of compensated and FP64 sums alone (1e-13 of the largest
partial sum), so 1e-9 of the largest acceleration is far above their difference.
Against FP64 each target has its own forward bound: a pair's term a_ij loses at
most 3 sqrt(3) u (|x_i| + |x_j|) / d_ij by the rounding of the coordinates (u =
2^-24; the term falls with the square of the distance and turns with it), 3 x
2^-22 by the approximate reciprocal root and 16 u by its other roundings and the
tile's sum of 128 terms is at most 128 u of the terms' magnitudes."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def to_system(nb, p, locked):
    if not locked:
        return nb.ParticleSystem(*[getattr(p, f).copy() for f in O.FIELDS])
    import torch

    s = nb.ParticleSystem.zeros(
        p.n, allocator=lambda k: torch.empty(k, dtype=torch.float64, pin_memory=True).numpy())
    for f in O.FIELDS:
        getattr(s, f)[:] = getattr(p, f)
    return s


def forward_bound(p, eps):
    u = 2.0 ** -24
    x = np.stack([p.x, p.y, p.z], axis=1)
    x = x - (p.m[:, None] * x).sum(0) / p.m.sum()
    r = np.linalg.norm(x, axis=1)
    d2 = ((x[:, None] - x[None]) ** 2).sum(2) + eps * eps
    np.fill_diagonal(d2, np.inf)
    d = np.sqrt(d2)
    term = p.m[None] / d2
    return (term * (3 * np.sqrt(3) * u * (r[:, None] + r[None]) / d + 3 * 2.0 ** -22 + 144 * u)).sum(1)


@pytest.mark.parametrize("n", [1, 2, 3, 127, 128, 129, 255, 256, 257, 1000, 1024, 1793, 2047, 2048])
@pytest.mark.parametrize("eps", [0.0, 0.01])
@pytest.mark.parametrize("locked", [False, True])
def test_all_pairs_plugin_equals_resident(cuda, n, eps, locked):
    p = O.preset_parallel("globular_cluster", max(n, 2), 4)
    p = O.Particles(*[getattr(p, f)[:n].copy() for f in O.FIELDS])
    s = to_system(cuda, p, locked)
    g = cuda.gravity_init(1.0, eps)
    with cuda.CudaContext() as c:
        a = cuda.n_body_sim_pro_gravity_compute_acceleration_cuda(s, g, c).copy()
        c.upload(s)
        exact = c.reference_acceleration(g, np.arange(n))
        c.compute_acceleration(g, cuda.Algorithm.ALL_PAIRS)
        b = c.download_accelerations()
    assert np.all(np.abs(a - exact) <= forward_bound(p, eps)[:, None])
    if n < 2048:  # (above, the resident path's tiles are the autotuner's)
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(b))


@pytest.mark.parametrize("n", [100, 2048, 20480, 20481])
@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("alpha", [0.0, 0.005])
def test_barnes_hut_plugin_equals_resident(cuda, n, locked, alpha):
    p = O.preset_parallel("globular_cluster", n, 4)
    s = to_system(cuda, p, locked)
    g = cuda.gravity_init(1.0, 0.01)
    with cuda.CudaContext(relative_opening=alpha) as c, cuda.CudaContext(relative_opening=alpha) as d:
        d.upload(s)
        for _ in range(2):  # the second call reads the first one's accelerations
            a = cuda.n_body_sim_pro_barnes_hut_compute_acceleration_cuda(s, g, c).copy()
            d.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
            np.testing.assert_array_equal(a, d.download_accelerations())


@pytest.mark.parametrize("locked", [False, True])
def test_errors_leave_the_context_usable(cuda, ctx, locked):
    p = O.preset_parallel("globular_cluster", 300, 4)
    g = cuda.gravity_init(1.0, 0.01)
    s = to_system(cuda, p, locked)
    s.y[211] = np.inf
    with pytest.raises(cuda.CudaError) as e:
        cuda.n_body_sim_pro_gravity_compute_acceleration_cuda(s, g, ctx)
    assert e.value.status == cuda.Status.INVALID_ARGUMENT
    s.y[211] = 0.5
    a = cuda.n_body_sim_pro_gravity_compute_acceleration_cuda(s, g, ctx)
    assert np.all(np.isfinite(a))
    import ctypes as C

    view, err = s.view(), cuda.Error()
    view.accelerations_z = C.POINTER(C.c_double)()
    status = cuda.library().n_body_sim_pro_gravity_compute_acceleration_cuda(
        C.byref(view), C.byref(g), ctx.handle, C.byref(err))
    assert status == cuda.Status.INVALID_ARGUMENT
