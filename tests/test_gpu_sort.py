"""The key sort at the edges of its tiles (4096 keys; up to one tile is sorted
by one block): permutation and sorted keys against numpy's stable sort, for
random keys, keys of few distinct values (long runs of equal digits, equal
128-bit keys in input order) and keys with constant digits. The keys are those
of positions, so that every case goes through the context's own entry points."""
import numpy as np
import pytest

from tandav_b200 import gravity as G

pytestmark = pytest.mark.gpu


def positions(kind, n, rng):
    pos = rng.random((3, n)) * 1000.0
    if kind == "few":                       # 27 points, thousands of times each
        pos = np.array([100.0, 500.0, 900.0])[rng.integers(0, 3, (3, n))]
    elif kind == "corner":                  # high digits equal for all keys
        pos = pos * 1e-3
    elif kind == "sorted":
        pos = np.sort(pos, axis=1)
    return pos


@pytest.mark.parametrize("kind", ["random", "few", "corner", "sorted"])
@pytest.mark.parametrize("n", [1, 2, 31, 257, 4095, 4096, 4097, 8192, 12289, 300_001])
def test_sort_tiles(kind, n):
    rng = np.random.default_rng(n)
    pos = positions(kind, n, rng)
    with G.GravityContext(max(n, 1024), float_bytes=8, periodic=True, boxsize=1000.0) as ctx:
        for _ in range(2):                  # the second call starts from the other buffers
            ctx.upload(pos, np.ones(n))
            ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
            ctx.peano_keys()
            keys = ctx.download(G.F_KEY)["key"]
            perm = ctx.sort_particles()
            out = ctx.download(G.F_KEY | G.F_ID | G.F_POS)
            order = np.lexsort((keys[:, 1], keys[:, 0]))      # stable
            np.testing.assert_array_equal(perm, order)
            np.testing.assert_array_equal(out["key"], keys[order])
            np.testing.assert_array_equal(out["id"], order)
            np.testing.assert_array_equal(out["pos"], pos[:, order])


@pytest.mark.parametrize("kind", ["random", "few", "corner"])
@pytest.mark.parametrize("n", [5119, 5121, (1 << 19) - 1, 1 << 19, (1 << 19) + 1])
def test_small_tiles(kind, n):
    """Tiles of 1024 keys below 2^19 + 1 keys, of 4096 above, in a context that
    has room for just these keys."""
    rng = np.random.default_rng(n)
    pos = positions(kind, n, rng)
    with G.GravityContext(n, float_bytes=8, periodic=True, boxsize=1000.0) as ctx:
        ctx.upload(pos, np.ones(n))
        ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
        ctx.peano_keys()
        keys = ctx.download(G.F_KEY)["key"]
        perm = ctx.sort_particles()
        out = ctx.download(G.F_KEY)
        order = np.lexsort((keys[:, 1], keys[:, 0]))
        np.testing.assert_array_equal(perm, order)
        np.testing.assert_array_equal(out["key"], keys[order])
