"""Every particle's acceleration in an ensemble against the FP64 sum of its system,
with the forward error bound of tests/test_small_plugin_gpu.py (its tiles of 128
sources bound the ensemble's of 64): softened, and unsoftened, where the kernel drops
the self pair, systems alone at the edges of tiles and in bundles."""
import numpy as np
import pytest

import oracle as O
from test_small_plugin_gpu import forward_bound

pytestmark = pytest.mark.gpu

SIZES = {"edges": [1, 2, 3, 63, 64, 65, 127, 128, 129, 1023, 1025, 2049, 2113],
         "equal": [300] * 400, "full": [4096, 4033], "unlike": list(range(1, 1200, 37))}


@pytest.mark.parametrize("name", list(SIZES))
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_accelerations_of_every_system(cuda, name, eps):
    sizes = SIZES[name]
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    mass = np.concatenate([rng.uniform(0.5, 1.5, k) / k for k in sizes])
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    s = cuda.ParticleSystem.from_arrays(rng.standard_normal((n, 3)), 0.1 * rng.standard_normal((n, 3)), mass)
    with cuda.CudaEnsemble() as e:
        e.upload(s, offsets)
        e.advance(cuda.gravity_init(1.0, eps), 1e-9, 1)  # (positions stay, but for their last bits)
        e.download(s)
    got = s.acc()
    for a, b in list(zip(offsets[:-1].astype(int), offsets[1:].astype(int)))[::max(1, len(sizes) // 40)]:
        p = O.Particles(*[getattr(s, f)[a:b].copy() for f in O.FIELDS])
        x = np.stack([p.x, p.y, p.z], axis=1)
        d = x[None] - x[:, None]
        r2 = (d * d).sum(2) + eps * eps
        np.fill_diagonal(r2, np.inf)
        exact = (p.m[None, :, None] * d / r2[:, :, None] ** 1.5).sum(1)
        assert np.all(np.abs(got[a:b] - exact) <= forward_bound(p, eps)[:, None])
