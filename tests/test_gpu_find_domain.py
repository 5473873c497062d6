"""tvg_find_domain's selection (tvg_domain.cu): the smallest sets, the sizes
around the second turn of a pass's loop (148 x 4 blocks of 1024 particles take
606,208 from particle 1 on), coordinates that are equal or zeros of either sign,
against the CPU restatement; the same numbers in both widths."""
import numpy as np
import pytest

import port
from tandav_b200 import gravity as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fsize", [4, 8])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 1024, 1025, 606_208, 606_209, 606_210, 2_000_003])
@pytest.mark.parametrize("kind", ["spread", "equal", "zeros"])
def test_find_domain_vs_restatement(kind, n, fsize):
    rng = np.random.default_rng(n)
    pos = rng.normal(0.0, 100.0, (3, n)) * np.array([[1.0], [1e-6], [1e6]])
    if kind == "equal":
        pos[0], pos[1] = -3.25, np.round(pos[1] * 1e4)
        pos[2, : n // 2] = 7.0
    if kind == "zeros":
        pos = rng.choice([-0.0, 0.0, -1e-30, 1e-30], (3, n))
        pos[:, -1] = (1.0, -2.0, 3.0)
    pos = pos.astype(port.ftype(fsize))
    origin, size = port.find_domain(pos, fsize)
    with G.GravityContext(n, float_bytes=fsize) as ctx:
        ctx.upload(pos, np.ones(n))
        if size == 0:                          # one particle: no domain, refused
            with pytest.raises(G.TvgError, match="BADINPUT"):
                ctx.find_domain()
            return
        for _ in range(2):                     # the second call starts from the first one's state
            o, s = ctx.find_domain()
            assert s == size and (o == origin).all()
