"""The sort of small systems (tiles of 1024 keys, then ranks among the tiles) at
the edges of its tiles and of its range, and the radix passes at the line between
their tile sizes: keys, permutation and root cube equal
the reference's bit for bit, with runs of equal keys in input order."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def to_system(nb, p):
    return nb.ParticleSystem(*[getattr(p, f).copy() for f in O.FIELDS])


@pytest.mark.parametrize("n", [2, 31, 1023, 1024, 1025, 8191, 9217, 98303, 98304, 98305, 449999, 450000])
@pytest.mark.parametrize("equal", [False, True])
def test_morton_order_of_small_systems(cuda, ctx, n, equal):
    p = O.preset_parallel("globular_cluster", n, 9)
    if equal:  # few distinct cells: long runs of equal keys across the tiles
        for f in ("x", "y", "z"):
            a = getattr(p, f)
            a[:] = np.clip(a, -1.0, 1.0)
            a[2:] = np.sign(a[2:]) * 0.5 + a[2:] * 1e-9
            a[0], a[1] = -1.0, 1.0
    ctx.upload(to_system(cuda, p))
    keys, perm, root = ctx.morton_order()
    ref_keys, ref_perm, ref_root = O.morton_order(p)
    np.testing.assert_array_equal(root, ref_root)
    np.testing.assert_array_equal(keys, ref_keys)
    np.testing.assert_array_equal(perm, ref_perm)
