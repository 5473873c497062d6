"""The plain walk's launch forms (tvg_walk_plain.cu). How many lanes share a
target follows from the number of active particles, and whether a warp's
targets walk together from how close they lie; neither may change a bit of a
target's force, potential or interaction count. So the walk over all
particles of a tree is compared, bit for bit, with walks over active lists of
its particles that take every other form. The FP32 form's rounded 1 / sqrt is
compared with the rounded operations over all significands."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tandav_b200 import build
from tandav_b200 import gravity as G
from tandav_b200 import ics

pytestmark = pytest.mark.gpu

N = 100_000          # the fewest targets that take one lane each in every part


@pytest.mark.parametrize("fsize,flags", [(4, 0), (8, 0), (4, G.CFG_POTENTIAL), (8, G.CFG_POTENTIAL)])
@pytest.mark.parametrize("use_bh", [True, False])
def test_forms_agree_bit_for_bit(fsize, flags, use_bh):
    # the box side is no float in the FP64 case, so both ways of wrapping run
    p = ics.random_box(N, box=1000.0 if fsize == 4 else 1000.1, seed=17, clumps=5)
    fields = G.F_GRAV_ACC | G.F_COST | (G.F_GRAV_POT if flags else 0)
    parts = G.WALK_GRAVITY | G.WALK_EWALD
    with G.GravityContext(N, float_bytes=fsize, periodic=True, boxsize=p.box, softening=p.softening,
                          flags=flags | G.CFG_FIX_SMALL_TOPNODES) as ctx:
        ctx.upload(p.pos, p.mass, last_acc=np.full(N, 3.0))
        ctx.set_domain((0.0, 0.0, 0.0), p.box)
        ctx.ewald_init()
        ctx.peano_keys()
        ctx.sort_particles()
        ctx.top_nodes()
        ctx.tree_build(exact_moments=True)
        ctx.zero_accel()
        ctx.walk(G.FORM_PLAIN, use_bh=use_bh, parts=parts)
        full = ctx.download(fields)
        rng = np.random.default_rng(3)
        lists = [np.arange(0, N - 1), np.arange(1, 45001), np.arange(44_999), np.arange(7, 8007),
                 np.arange(50_000, 57_999), np.arange(3, 20), np.arange(0, N, 100),
                 np.sort(rng.choice(N, 12_001, replace=False))]
        for active in lists:
            ctx.set_active(None)
            ctx.zero_accel()
            ctx.set_active(active)
            ctx.walk(G.FORM_PLAIN, use_bh=use_bh, parts=parts)
            got = ctx.download(fields)
            for k in full:
                np.testing.assert_array_equal(got[k][..., active], full[k][..., active],
                                              err_msg=f"{k}, {len(active)} active")


def test_inv_sqrt_equals_the_rounded_operations(tmp_path):
    nvcc = shutil.which("nvcc") or build.nvcc()
    exe = tmp_path / "inv_sqrt_check"
    src = Path(__file__).with_name("inv_sqrt_check.cu")
    subprocess.run([nvcc, *build.ARCH, "-O3", "-fmad=false", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True)
    assert int(out.stdout) == 0
