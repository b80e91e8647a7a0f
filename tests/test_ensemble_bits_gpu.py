"""A system of an ensemble evolves to the same bits whatever it is bundled with:
how many warps serve it depends on its neighbours, on the number of systems and on
the tuned block shape, and with them where a target tile's sources are cut between
two warps.  Sizes at the edges of tiles (64 particles), of slots (4096) and where
runs of tile pairs are unequal; masses that differ by up to 1e12 from tile to tile (a
star among dust), where compensated sums in another grouping round differently."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 63, 64, 65, 129, 192, 300, 448, 640, 700, 833, 1025, 1344, 2047, 2113, 2500, 3000, 4033, 4096]


def evolve(nb, systems, eps):
    """The final state of each of (pos, vel, mass)."""
    pos, vel, mass = (np.concatenate(a) for a in zip(*systems))
    offsets = np.concatenate([[0], np.cumsum([len(s[2]) for s in systems])]).astype(np.uint64)
    s = nb.ParticleSystem.from_arrays(pos, vel, mass)
    with nb.CudaEnsemble() as e:
        e.upload(s, offsets)
        e.advance(nb.gravity_init(1.0, eps), 1e-3, 3)
        e.download(s)
    out = np.stack([s.x, s.y, s.z, s.vx, s.vy, s.vz, s.ax, s.ay, s.az])
    return [out[:, a:b] for a, b in zip(offsets[:-1].astype(int), offsets[1:].astype(int))]


@pytest.fixture(scope="module")
def systems():
    rng = np.random.default_rng(8)
    return [(rng.standard_normal((k, 3)), 0.1 * rng.standard_normal((k, 3)),
             np.repeat(10.0 ** rng.uniform(-12, 0, -(-k // 64)), 64)[:k]) for k in SIZES]


@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_bits_do_not_depend_on_the_bundle(cuda, systems, eps):
    alone = [evolve(cuda, [s], eps)[0] for s in systems]
    for copies in (1, 3):  # among unlike neighbours
        order = np.random.default_rng(copies).permutation(len(systems) * copies) % len(systems)
        for k, got in zip(order, evolve(cuda, [systems[k] for k in order], eps)):
            np.testing.assert_array_equal(got, alone[k], err_msg=f"{copies} of {SIZES[k]}")
    for k, n in enumerate(SIZES):  # among its like, as many as fill an item for each of 148 SMs
        tiles = -(-n // 64)
        for got in evolve(cuda, [systems[k]] * (148 * min(32, 64 // tiles)), eps)[::37]:
            np.testing.assert_array_equal(got, alone[k], err_msg=f"full items of {n}")
