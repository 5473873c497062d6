"""The group form's two Ewald tables as the device holds them, through the walk:
the force of one particle on massless ones, against the FP64 Ewald sum. A compact
set of targets takes the expansion of the 33-node record (value, first and second
derivatives at the group centre), a set spread over the box each target's own
lookup of the 41-node record."""
import numpy as np
import pytest

from tandav_b200 import gravity as G

pytestmark = pytest.mark.gpu

L = 100.0


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("fsize", [4, 8])
def test_force_of_one_particle(fsize, spread):
    """Bound, in units of G m / L^2: the pair force in FP32 (4e-7 of at most
    25, targets keep 0.2 L from the source) and the correction: compact (within
    L / 400), value and gradient of the record (5e-7, 4e-5 x 4 / 400), its second
    derivatives (4e-3 x 100 / 400^2 / 2) and the expansion's remainder
    (1000 / 400^3 / 6): 6e-6 in all; spread, the value alone: 2e-6."""
    rng = np.random.default_rng(5)
    bound = 4e-7 * 25 + (2e-6 if spread else 6e-6)
    n, worst = 33, 0.0
    for _ in range(24):
        src = rng.uniform(0.0, L, 3)
        while True:
            c = rng.uniform(0.02 * L, 0.98 * L, (3, n - 1 if spread else 1))
            d = np.abs(c - src[:, None])
            far = np.sqrt((np.minimum(d, L - d) ** 2).sum(0)) > 0.21 * L
            if far.sum() >= min(20, c.shape[1]):
                break
        c = np.where(far, c, c[:, far][:, :1])
        pos = np.empty((3, n))
        pos[:, 0] = src
        pos[:, 1:] = c if spread else c + rng.uniform(-1.0, 1.0, (3, n - 1)) * L / 400 / np.sqrt(3)
        if spread:                             # (targets moved together: no two at one place)
            pos[:, 1:] += rng.uniform(-1e-3, 1e-3, (3, n - 1)) * L
        mass = np.full(n, 1e-18)
        mass[0] = 1.0
        with G.GravityContext(n, float_bytes=fsize, periodic=True, boxsize=L, gravity=1.0, softening=1e-3,
                              open_bh=1e-12, vector_size=8) as ctx:
            ctx.set_domain((0.0, 0.0, 0.0), L)
            ctx.ewald_init()
            ctx.set_ewald_opening(1e-12, 1e-12)
            ctx.upload(pos, mass)
            ctx.peano_keys()
            targets = np.flatnonzero(ctx.sort_particles() != 0)
            ctx.top_nodes()
            ctx.tree_build(exact_moments=False)
            ctx.set_active(targets)
            ctx.walk(G.FORM_GROUP, use_bh=True, parts=G.WALK_GRAVITY | G.WALK_EWALD)
            direct, tree, _ = ctx.forcetest(targets)
        worst = max(worst, np.abs(tree - direct).max() * L * L)
    assert worst < bound
