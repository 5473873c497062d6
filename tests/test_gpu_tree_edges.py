"""The tree build where its searches and warps have edges: particle counts
around the 64-byte blocks and 8-byte words of the level searches, a single
top node and many, a dense clump (node ends thousands of blocks away, exact
sums over nodes of more than 256 and more than 8192 particles), against the
oracle's sequential build, every field bit for bit."""
import numpy as np
import pytest

import port
from pipeline import assert_struct_equal
from tandav_b200 import gravity as G
from test_gpu_parity import TOP_FIELDS, TREE_FIELDS, gpu_pipeline, make_ctx

pytestmark = pytest.mark.gpu


def clumps(n, seed, one_cell):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 240.0 if one_cell else 1000.0, (3, n))
    m = n // 2
    pos[:, :m] = np.array([[120.3], [77.7], [201.1]]) + rng.normal(0.0, 0.5, (3, m))
    return pos, rng.uniform(0.5, 1.5, n)


@pytest.mark.parametrize("one_cell", [False, True])
@pytest.mark.parametrize("fsize", [4, 8])
@pytest.mark.parametrize("n,vsize", [(9, 4), (63, 8), (64, 8), (65, 8), (127, 16), (129, 64), (257, 1),
                                     (4095, 64), (4097, 32), (40_000, 64)])
def test_tree_edges_vs_oracle(n, vsize, fsize, one_cell):
    pos, mass = clumps(n, n, one_cell)
    ft = port.ftype(fsize)
    pos_f = pos.astype(ft)
    std, rev = port.peano_keys(pos_f, np.zeros(3), 1000.0, fsize)
    perm_o = port.sort_keys(std)
    pos_s, mass_s = pos_f[:, perm_o], mass.astype(ft)[perm_o]
    top_o = port.top_nodes(std[perm_o], pos_s, np.zeros(3), 1000.0, fsize)
    tree_o, top_o, parent_o = port.tree_build(rev[perm_o], pos_s, mass_s, 1000.0, top_o, fsize,
                                              vector_size=vsize)
    with make_ctx(n, fsize, box=1000.0, softening=0.1, vector_size=vsize) as ctx:
        perm, _, tree, top = gpu_pipeline(ctx, pos, mass, np.zeros(3), 1000.0, exact=True)
        parent = ctx.download(G.F_TREE_PARENT)["tree_parent"]
    assert np.array_equal(perm, perm_o)
    assert_struct_equal(top, top_o, TOP_FIELDS, "topnodes")
    assert_struct_equal(tree, tree_o, TREE_FIELDS, "tree")
    assert np.array_equal(parent, parent_o)


@pytest.mark.parametrize("n", [3000, 65_535, 65_536, 65_537])
def test_tree_at_capacities(n):
    """The build's scans run over the capacity (2 c + 4097 items), the active
    set's over n: with one launch up to 16 tiles of 4096 items, two up to 2048,
    and a scan of the sums beyond. The same particles give the same tree, the
    same forces and the same window groups at capacities on both sides."""
    pos, mass = clumps(n, 5, False)
    caps = [c for c in (n, 30_719, 30_720, 4_192_255, 4_192_256) if c >= n]
    active = np.arange(0, n, 3)
    out = []
    for cap in caps:
        with G.GravityContext(cap, softening=1.0, vector_size=16, flags=G.CFG_QUADRUPOLE) as ctx:
            ctx.upload(pos.astype(np.float32), mass.astype(np.float32))
            ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
            ctx.force_step(form=G.FORM_GROUP, use_bh=True, parts=G.WALK_GRAVITY)
            ctx.set_active(active)
            ctx.walk(G.FORM_GROUP, use_bh=True, parts=G.WALK_GRAVITY)
            tree, top = ctx.download_tree()
            d = ctx.download(G.F_GRAV_ACC | G.F_COST | G.F_TREE_PARENT)
            out.append((tree, top, d["cost"], d["tree_parent"], d["grav_acc"]))
    for tree, top, cost, parent, acc in out[1:]:
        np.testing.assert_array_equal(tree, out[0][0])
        np.testing.assert_array_equal(top, out[0][1])
        np.testing.assert_array_equal(cost, out[0][2])
        np.testing.assert_array_equal(parent, out[0][3])
        np.testing.assert_array_equal(acc, out[0][4])
