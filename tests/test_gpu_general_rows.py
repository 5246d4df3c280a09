"""General panel pairs of a real wavenumber (k_general: one thread per pair and Gauss
node, Hankel functions from the table of hankel_u.cuh) where they can go wrong: the
lowest and highest quadrature orders (pairs per CTA 64 and 4), meshes with fewer pairs
than a CTA takes and with a remainder, lines and arcs in one mesh, and arguments across
the table's upper end.  Against the oracle's GalerkinBuilder restatement at
the usual 1e-12 relative Frobenius (at the largest arguments, x = ks r up to 1200, the
rounding of x alone moves the phase by x eps = 3e-13)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api, geometry  # noqa: E402
from oracle import oracle as O  # noqa: E402


def half_disc(n):
    """A half circle of arcs closed by line panels."""
    kinds, par = geometry.circle(0.3, 2 * n)
    flat = np.array(geometry.split_line((-0.3, 0.0), (0.3, 0.0), n))
    par = par[:n].copy()
    par[n - 1, 4] = np.pi
    # end points of the straight part exactly where the arcs end
    e0 = par[0]
    flat[-1, 2:4] = (e0[2] * np.cos(e0[3]), e0[2] * np.sin(e0[3]))
    flat[0, 0:2] = (0.3 * np.cos(np.pi), 0.3 * np.sin(np.pi))
    return (np.concatenate([kinds[:n], np.zeros(n, np.int32)]).astype(np.int32), np.concatenate([par, flat]))


CASES = {
    "order2": (lambda: geometry.circle(0.25, 13), 2, 3.3, 7.0),
    "order3_lines": (lambda: geometry.polygon(*geometry.star_polygon(9, seed=1), 19), 3, 3.3, 7.0),
    "order32": (lambda: geometry.circle(0.25, 7), 32, 2.2, 9.0),
    "order17_lines": (lambda: geometry.polygon(*geometry.star_polygon(5, seed=4), 11), 17, 2.2, 9.0),
    "four_panels": (lambda: geometry.circle(0.25, 4), 11, 1.1, 4.0),
    "three_panels": (lambda: geometry.circle(0.25, 3), 7, 1.1, 4.0),
    "mixed_panels": (lambda: half_disc(6), 11, 4.0, 5.0),
    "large_arguments": (lambda: geometry.circle(1.0, 24), 11, 600.0, 1.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_layers_match_the_oracle(name):
    make, order, k, c = CASES[name]
    kinds, par = make()
    gb = api.GalerkinBuilder(api.BuilderData((kinds, par), order=order))
    ob = O.Builder(kinds, par, order)
    for d in (0, 1, 2):
        gb.assembleDense(k, c, d=d)
        ref = ob.assemble(k, c, O.LAYER_ALL, d)
        for got, key in ((gb.getDoubleLayer, "K"), (gb.getHypersingular, "W"), (gb.getSingleLayer, "V")):
            for t in range(d + 1):
                err = np.linalg.norm(got(t) - ref[key][t]) / np.linalg.norm(ref[key][t])
                assert err <= 1e-12, (name, d, key, t, err)
