"""The octree build at the edges of its blocks and with the smallest and largest
buckets: the interaction-list walk (walk ids, consecutive siblings) and the
stackless walk (depth-first order) traverse the same tree through different
records, and both stay within the reference's own bound of the direct sum
(tests/numerical/barnes_hut_test.c: theta 0.3, rms below 1e-2)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def to_system(nb, p):
    return nb.ParticleSystem(*[getattr(p, f).copy() for f in O.FIELDS])


@pytest.mark.parametrize("n", [2, 3, 9, 33, 1023, 1024, 1025, 1026, 2049, 3073])
@pytest.mark.parametrize("leaf", [1, 16, 64])
@pytest.mark.parametrize("order", [1, 2])
def test_walks_agree_on_the_tree(cuda, n, leaf, order):
    s = to_system(cuda, O.preset_parallel("globular_cluster", n, 3))
    g = cuda.gravity_init(1.0, 0.01)
    results, counts = [], []
    for walk in (0, 1):
        with cuda.CudaContext(theta=0.3, leaf_capacity=leaf, multipole_order=order) as c:
            c.set_walk(walk)
            results.append(cuda.n_body_sim_pro_barnes_hut_compute_acceleration_cuda(s, g, c).copy())
            st = c.stats()
            counts.append([st[k] for k in ("node_count", "leaf_count", "maximum_depth",
                                           "accepted_approximations", "exact_interactions")])
    assert counts[0] == counts[1]
    assert counts[0][0] >= counts[0][1] >= 1
    # the same terms in another order, FP32 partial sums of at most 64 terms
    rms = np.sqrt(np.mean(results[0] ** 2))
    assert np.sqrt(np.mean((results[0] - results[1]) ** 2)) <= 2e-6 * rms
    with cuda.CudaContext() as c:
        c.upload(s)
        exact = c.reference_acceleration(g, np.arange(n))
    assert np.sqrt(np.sum((results[1] - exact) ** 2) / np.sum(exact ** 2)) < 1e-2


@pytest.mark.parametrize("n", [75776, 75777, 227328, 227329])
@pytest.mark.parametrize("order, alpha", [(1, 0.0), (1, 0.005), (2, 0.0)])
def test_walk_forms_take_the_same_decisions(cuda, n, order, alpha):
    """Either side of the lines between the list walk's register forms: the same
    cells and particles as the stackless walk, the same sums to FP32 rounding."""
    s = to_system(cuda, O.preset_parallel("globular_cluster", n, 3))
    g = cuda.gravity_init(1.0, 0.01)
    results, counts = [], []
    for walk in (0, 1):
        with cuda.CudaContext(theta=0.7, multipole_order=order, relative_opening=alpha) as c:
            c.set_walk(walk)
            c.upload(s)
            for _ in range(2 if alpha > 0.0 else 1):
                c.compute_acceleration(g, cuda.Algorithm.BARNES_HUT)
            results.append(c.download_accelerations())
            st = c.stats()
            counts.append([st["accepted_approximations"], st["exact_interactions"]])
    if alpha == 0.0:
        assert counts[0] == counts[1]
    else:  # the first evaluations' roundings move the second's tolerances
        assert abs(counts[0][0] - counts[1][0]) <= 1e-6 * counts[1][0]
    rms = np.sqrt(np.mean(results[0] ** 2))
    bar = 2e-6 if alpha == 0.0 else 2e-5
    assert np.sqrt(np.mean((results[0] - results[1]) ** 2)) <= bar * rms
