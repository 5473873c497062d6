"""The 33-node record as the group form's lookup uses it: the three entries of
d3T with one x, y or none and three z from the zero trace (ewald_third), the others
from the table, against direct lattice sums at random points of the octant."""
import numpy as np

import ewald_taylor as TT
import port

N = 33
G = 2 * (N - 1)


def test_lookup_against_lattice_sums():
    """Value within 6e-7 of |T| and gradient within 5e-5 of its largest
    component at 60 points (third-order expansion over half a node spacing, whose
    remainder is largest near the corners of the octant)."""
    rng = np.random.default_rng(12)
    for x in rng.uniform(0.0, 0.5, (60, 3)):
        node = np.rint(x * G).astype(int)
        t = TT.lookup(TT.tensors(TT.record(node, N)))
        assert all(abs(t[3][a, b, 0, 0] + t[3][a, b, 1, 1] + t[3][a, b, 2, 2]) < 1e-12
                   for a, b in ((0, 1), (0, 2), (1, 2)))
        val, grad, _ = TT.evaluate_tensors(t, x * G - node)
        exact = port.ewald_force(x)[0]
        assert np.abs(val - exact).max() <= 6e-7 * max(np.linalg.norm(exact), 1e-2)
        e, jac = 1e-4 / G, np.zeros((3, 3))
        for b in range(3):
            d = np.zeros(3)
            d[b] = e
            jac[:, b] = (port.ewald_force(x + d)[0] - port.ewald_force(x - d)[0]) / (2 * e * G)
        assert np.abs(grad - jac).max() <= 5e-5 * max(np.abs(jac).max(), 1e-3)
