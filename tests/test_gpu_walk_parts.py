"""Walks whose groups are not split, the kernels of large runs, against walks
of a few of the same groups in 2 to 32 parts. That the former are not split is read
off the launches: a walk that may split launches a kernel more for each of its two
walks (k_walk_sum, k_ewald_sum)."""
import numpy as np
import pytest

from tandav_b200 import gravity as G
from tandav_b200 import ics

pytestmark = pytest.mark.gpu


def launches(ctx, parts):
    before = ctx.launch_count()
    ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
    return ctx.launch_count() - before


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("flags", [0, G.CFG_QUADRUPOLE])
def test_unsplit_groups(periodic, flags):
    """1.25M particles make 19,532 groups of 64, one part each; windows of the
    same order make few groups of the same particles. Counts equal; forces equal up
    to the order of FP32 sums carried in FP64 (1e-4 of the largest component, as for
    the split groups among themselves)."""
    parts = G.WALK_GRAVITY | (G.WALK_EWALD if periodic else 0)

    def context(n):
        p = ics.random_box(n, box=1000.0, seed=91, clumps=6)
        ctx = G.GravityContext(n, periodic=periodic, boxsize=1000.0 if periodic else 0.0,
                               softening=p.softening, flags=flags, open_rel=8e-3)
        ctx.upload(p.pos, p.mass, last_acc=np.full(n, 3.0))
        ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
        ctx.set_ewald_opening(1e-2)
        ctx.force_step(form=G.FORM_GROUP, use_bh=False, parts=parts)
        return ctx

    with context(5000) as ctx:                       # 79 groups: 32 parts
        split = launches(ctx, parts)
    n = 1_250_000
    with context(n) as ctx:
        assert launches(ctx, parts) == split - (2 if periodic else 1)
        full = ctx.download(G.F_GRAV_ACC | G.F_COST)
        acc, cost = full["grav_acc"].astype(np.float64), full["cost"]
        last = (n - 1) // 64
        for windows in (np.arange(1), np.arange(3, 200, 2), np.arange(0, 2300), np.arange(last, last + 1)):
            active = (64 * windows[:, None] + np.arange(64)[None]).reshape(-1)
            active = active[active < n]
            ctx.set_active(active)
            ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
            got = ctx.download(G.F_GRAV_ACC | G.F_COST)
            np.testing.assert_array_equal(got["cost"][active], cost[active])
            d = np.abs(got["grav_acc"].astype(np.float64)[:, active] - acc[:, active])
            assert d.max() < 1e-4 * np.abs(acc).max()
            assert ctx.walk_counters()[0] == cost[active].astype(np.float64).sum()
