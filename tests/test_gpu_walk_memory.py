"""The group walks' memory for the sums of split groups: as much as the
context's groups can use, grown when another walk needs more, and a walk that
cannot have it goes on with one part a group."""
import numpy as np
import pytest
import torch

from tandav_b200 import gravity as G
from tandav_b200 import ics

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free():
    return torch.cuda.mem_get_info()[0]


def context(n_side, fsize=4):
    p = ics.zeldovich_box(n_side=n_side, seed=5) if n_side else ics.hernquist(3001, seed=5)
    per = n_side > 0
    ctx = G.GravityContext(p.n, float_bytes=fsize, periodic=per, boxsize=p.box if per else 0.0,
                           softening=p.softening, vector_size=32, open_rel=8e-3)
    ctx.upload(p.pos, p.mass, last_acc=np.full(p.n, 0.02 if per else 1e4))
    if per:
        ctx.set_domain((0.0, 0.0, 0.0), p.box)
        ctx.ewald_init()
        ctx.set_ewald_opening(1e-2)
    else:
        ctx.find_domain()
    return ctx, G.WALK_GRAVITY | (G.WALK_EWALD if per else 0)


# 32 bytes a target slot of at most 32 parts of each 64-particle group, and at
# most 16 items for each of 2368 warps; per-target images 24 bytes of at most 4736
# items; beside them the group form's two Ewald tables (12 MB) and the
# allocator's rounding
@pytest.mark.parametrize("n_side,fsize,most", [(0, 4, 3), (32, 4, 34), (64, 8, 8), (64, 4, 78)])
def test_first_step_takes_what_its_groups_can_use(n_side, fsize, most):
    for measured in (False, True):              # the first run also loads the kernels
        ctx, parts = context(n_side, fsize)
        before = free()
        ctx.force_step(form=G.FORM_GROUP, use_bh=False, parts=parts)
        used = before - free()
        ctx.close()
    assert used <= (most + (16 if n_side else 4)) * MB


def test_walk_without_memory_for_the_parts():
    ctx, parts = context(64)
    ctx.peano_keys()
    ctx.sort_particles()
    ctx.top_nodes()
    ctx.tree_build(exact_moments=False)
    fields = G.F_GRAV_ACC | G.F_COST
    ctx.set_active(np.arange(64))               # everything but the full walk's sums is allocated here
    ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
    ctx.set_active(None)
    torch.cuda.empty_cache()
    hold = torch.empty(free() // (2 * MB) * 2 * MB - 40 * MB, dtype=torch.uint8, device="cuda")
    before = free()
    ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
    assert before - free() < 8 * MB
    one = ctx.download(fields)
    del hold
    torch.cuda.empty_cache()
    before = free()
    ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
    assert before - free() > 40 * MB             # more than was left before
    split = ctx.download(fields)
    ctx.close()
    np.testing.assert_array_equal(one["cost"], split["cost"])
    a, b = (d["grav_acc"].astype(np.float64) for d in (one, split))
    # FP32 sums of at most 256 entries carried in FP64, as for the split groups
    assert np.abs(a - b).max() < 1e-4 * np.abs(a).max()


def test_captured_step_is_dropped_when_the_memory_moves():
    """A captured step whose groups are not split holds the memory of the groups
    with per-target images; a walk of a list needs more. The steps after it are
    captured anew and give the force that steps without that walk give (up to
    nodes at the edge of the criterion: |a_old| of the list's particles comes from
    walks in other parts)."""
    n, parts = 1_250_000, G.WALK_GRAVITY | G.WALK_EWALD
    p = ics.random_box(n, box=1000.0, seed=3, clumps=6)
    out = []
    for with_list in (False, True):
        with G.GravityContext(n, periodic=True, boxsize=1000.0, softening=p.softening, open_rel=8e-3) as ctx:
            ctx.upload(p.pos, p.mass, last_acc=np.full(n, 3.0))
            ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
            ctx.ewald_init()
            ctx.set_ewald_opening(1e-2)
            for _ in range(3):                 # direct, captured, captured in the other buffers
                ctx.step_graph(parts=parts)
            if with_list:
                before = free()
                ctx.set_active(np.arange(64 * 100))
                ctx.walk(G.FORM_GROUP, use_bh=False, parts=parts)
                assert before - free() > 8 * MB
            for _ in range(4):
                ctx.step_graph(parts=parts)
            d = ctx.download(G.F_GRAV_ACC | G.F_ID)
            out.append(d["grav_acc"].astype(np.float64)[:, np.argsort(d["id"])])
    assert np.abs(out[1] - out[0]).max() < 1e-2 * np.abs(out[0]).max()
