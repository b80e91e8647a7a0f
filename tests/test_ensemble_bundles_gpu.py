"""The ensemble kernel where its split of the work can go wrong: systems at the
edges of tiles and slots, bundles of equal and of unlike sizes, more and fewer
systems than SMs, and runs of tile pairs that share a tile of targets.  Each
system against the per-system launches of the same library (other kernels):
FP32 pair sums in other tiles, a few 1e-7 of the accelerations, which over two
steps of 1e-3 move a velocity by about 1e-9 of them; 1e-7 leaves the closest
pairs of the smallest systems (accelerations of some 1e2) a factor of ten."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = {
    "edges": [1, 2, 63, 64, 65, 127, 128, 129, 1023, 1024, 1025, 2047, 2048, 2049, 2111, 2112, 2113,
              3000, 4032, 4033, 4095, 4096],
    "equal": [64] * 600,
    "tiles_21": [1344] * 160,
    "unlike": list(range(1, 4097, 23)),
    "few": [700, 650, 90],
}


@pytest.mark.parametrize("name", list(SIZES))
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_bundles_match_per_system_launches(cuda, name, eps):
    sizes = SIZES[name]
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    pos = rng.standard_normal((n, 3))
    vel = 0.1 * rng.standard_normal((n, 3))
    mass = np.concatenate([np.full(k, 1.0 / k) for k in sizes])
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    g = cuda.gravity_init(1.0, max(eps, 0.0))
    got = []
    for per_system in (False, True):
        s = cuda.ParticleSystem.from_arrays(pos, vel, mass)
        with cuda.CudaEnsemble() as e:
            e.upload(s, offsets)
            e.advance(g, 1e-4 if eps == 0.0 else 1e-3, 2, one_launch_per_system=per_system)
            e.download(s)
        got.append(np.stack([s.x, s.y, s.z, s.vx, s.vy, s.vz]))
    assert np.all(np.isfinite(got[0]))
    # unsoftened pairs can be arbitrarily close: all but the closest few
    off = np.abs(got[0] - got[1])
    if eps > 0.0:
        assert np.max(off) <= 1e-7
    else:
        assert np.mean(off > 1e-7) < 1e-3
