"""The plain walk where its reads have edges. Without
TVG_CFG_FIX_SMALL_TOPNODES a small top node's particles are taken from its
Target on, a running node count: with bundles of one particle the nodes
outnumber the particles and Target passes the last of them. What lies there
counts as a massless particle at the origin, whatever the capacity and whatever
an earlier, larger upload left behind. Where the box side is a float, FP32 bundles
that reach the half-box plane wrap in float (gravity_run); where it is not, they
take the general form."""
import numpy as np
import pytest

import port
from pipeline import oracle_ewald_tables, oracle_pipeline
from tandav_b200 import gravity as G
from test_gpu_parity import gpu_pipeline, reference_table, walks

pytestmark = pytest.mark.gpu

BOX = 1000.0


def clump_and_singles(n, singles):
    """n - singles particles of a clump in the level-2 cell with the largest
    key, and single particles in cells of smaller keys, whose top nodes follow."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, BOX, (3, 4000))
    std, _ = port.peano_keys(pos, np.zeros(3), BOX, 8)
    cell = (std[:, 0] >> np.uint64(58)).astype(int)
    high = pos[:, cell == 63][:, :1]
    out = high + rng.normal(0.0, 0.5, (3, n))
    for k in range(singles):
        out[:, k] = pos[:, cell == 2 * k + 1][:, 0]
    return out, rng.uniform(0.5, 1.5, n)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("use_bh", [True, False])
@pytest.mark.parametrize("fsize", [4, 8])
def test_small_top_nodes_past_the_last_particle(fsize, use_bh, periodic):
    """Against the oracle, which reads the same places of arrays that end in
    zeros: counts, force and potential bit for bit."""
    n, ft = 300, port.ftype(fsize)
    pos, mass = clump_and_singles(n, 20)
    parts = G.WALK_GRAVITY | (G.WALK_EWALD if periodic else 0)
    fields = G.F_GRAV_ACC | G.F_COST | G.F_GRAV_POT
    out = []
    for cap in (n, n + 1, 4 * n):
        with G.GravityContext(cap, float_bytes=fsize, periodic=periodic, boxsize=BOX if periodic else 0.0,
                              softening=0.1, vector_size=1, flags=G.CFG_POTENTIAL) as ctx:
            def load(p, m):
                ctx.upload(p, m)
                ctx.set_domain((0.0, 0.0, 0.0), BOX)
                ctx.peano_keys()
                ctx.sort_particles()
                ctx.top_nodes()
                ctx.tree_build(exact_moments=True)
            if periodic:
                ctx.upload_ewald_table(*reference_table(fsize))
            if cap > 2 * n:          # leave other particles past the last one
                load(np.random.default_rng(1).uniform(1.0, BOX - 1.0, (3, cap)), np.full(cap, 1e3))
            load(pos, mass)
            ctx.zero_accel()
            ctx.walk(G.FORM_PLAIN, use_bh=use_bh, parts=parts)
            out.append(ctx.download(fields | G.F_POS | G.F_MASS))
            tree, top = ctx.download_tree()
    small = top[top["Npart"] == 1]
    assert len(small) == 20 and (small["Target"] >= n).all()
    for d in out[1:]:
        for k in out[0]:
            np.testing.assert_array_equal(d[k], out[0][k], err_msg=k)
    pad = int(small["Target"].max()) + 2
    x, m = np.zeros((3, n + pad), ft), np.zeros(n + pad, ft)
    x[:, :n], m[:n] = out[0]["pos"], out[0]["mass"]
    prm = port.WalkParams(gravity=G.GRAVITY, softening=0.1, domain_size=BOX, boxsize=BOX if periodic else 0.0,
                          open_bh=0.25, open_rel=0.005, use_bh=int(use_bh), vector_size=1)
    a, cost, pot = port.walk("gravity", x, m, np.zeros(n + pad), top, tree, prm, fsize=fsize, potential=True)
    acc, cost, pot = a[:, :n].astype(ft), cost[:n].astype(ft), pot[:n].astype(ft)
    if periodic:
        tabs = [(t.astype(np.float64) / (BOX if k == 3 else BOX * BOX)).astype(ft)
                for k, t in enumerate(reference_table(fsize))]
        e, ce, pe = port.walk("ewald", x, m, np.zeros(n + pad), top, tree, prm, tabs, fsize=fsize, potential=True)
        acc = (acc.astype(np.float64) + e[:, :n]).astype(ft)
        cost = (cost + ce[:n].astype(ft)).astype(ft)
        pot = (pot.astype(np.float64) + pe[:n]).astype(ft)
    np.testing.assert_array_equal(out[0]["cost"], cost)
    np.testing.assert_array_equal(out[0]["grav_acc"], acc)
    np.testing.assert_array_equal(out[0]["grav_pot"], pot)


@pytest.mark.parametrize("box", [1000.0, 1000.1])
def test_bundles_across_the_half_box_plane(box):
    """FP32 boxes whose bundles of up to 64 particles are wide enough for many of
    them to straddle a target's half-box plane: force and count bit for bit."""
    rng = np.random.default_rng(8)
    n = 4003
    pos = rng.uniform(0.0, 999.9, (3, n)).astype(np.float32)
    mass = rng.uniform(0.5, 1.5, n)
    o = oracle_pipeline(pos, mass, np.zeros(3), box, 4, box=box, softening=2.0,
                        ewald=oracle_ewald_tables(4, box))
    with G.GravityContext(n, periodic=True, boxsize=box, gravity=43007.1, softening=2.0) as ctx:
        perm, _, _, _ = gpu_pipeline(ctx, pos, mass, np.zeros(3), box)
        assert np.array_equal(perm, o["perm"])
        bh, _, rel = walks(ctx, True, 4)
    for name, got in (("bh", bh), ("rel", rel)):
        np.testing.assert_array_equal(got["cost"], o[name + "_cost"])
        np.testing.assert_array_equal(got["grav_acc"], o[name + "_gacc"])
