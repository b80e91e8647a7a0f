"""Launch shapes between those of the neighbouring files: clusters of 3, 5, 6 and 7
blocks of the small all-pairs kernels and of the training epoch, cooperative epochs
of 9 to 31 blocks, plugin calls at the largest system that is staged (16,384) and
one more, and unaligned arrays.  References and tolerances are those files'."""
import numpy as np
import pytest

import oracle as O
import test_correction_epoch_gpu as epochs
import test_small_plugin_gpu as plugin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [513, 700, 768, 1025, 1280, 1281, 1536, 1537, 1792])
@pytest.mark.parametrize("eps", [0.0, 0.01])
@pytest.mark.parametrize("locked", [False, True])
def test_all_pairs_clusters(cuda, n, eps, locked):
    plugin.test_all_pairs_plugin_equals_resident(cuda, n, eps, locked)


@pytest.mark.parametrize("n", [16383, 16384, 16385])
@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("alpha", [0.0, 0.005])
def test_staged_barnes_hut(cuda, n, locked, alpha):
    plugin.test_barnes_hut_plugin_equals_resident(cuda, n, locked, alpha)


@pytest.mark.parametrize("samples, batch", [(1000, 384), (1500, 640), (1800, 768), (2100, 896),
                                            (2600, 1152), (4700, 2048), (9000, 3968)])
def test_epoch_blocks(cuda, samples, batch):
    epochs.test_epoch_equals_its_steps(cuda, samples, batch)


@pytest.mark.parametrize("n", [300, 2047, 3000])
@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("algorithm", ["gravity", "barnes_hut"])
def test_unaligned_arrays(cuda, n, locked, algorithm):
    """Arrays 4 bytes off their alignment give what aligned ones do."""
    import torch

    p = O.preset_parallel("globular_cluster", n, 4)
    g = cuda.gravity_init(1.0, 0.01)
    raw = [torch.empty(8 * n + 4, dtype=torch.uint8, pin_memory=locked) for _ in O.FIELDS]
    s = cuda.ParticleSystem(*[r.numpy()[4:].view(np.float64) for r in raw])
    for f in O.FIELDS:
        getattr(s, f)[:] = getattr(p, f)
    assert not s.x.flags.aligned
    call = getattr(cuda, f"n_body_sim_pro_{algorithm}_compute_acceleration_cuda")
    with cuda.CudaContext() as c:
        got = call(s, g, c)
        np.testing.assert_array_equal(got, call(plugin.to_system(cuda, p, False), g, c))
