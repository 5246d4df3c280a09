"""The grid kernel of the field at real k (Hankel table, FP32 look at the panels before the
FP64 tests) where it can go wrong: fewer nodes than a tile and a remainder of one, grids of
fewer points than a CTA, points in the segments of long arcs, near and far from a mesh of
one scale, arguments beyond the table (kappa r up to 1500), a mesh away from the
origin (the FP32 coordinates lose digits there).  Against the oracle at the field tests'
1e-8 of the field's maximum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api, geometry  # noqa: E402
from oracle import oracle as O  # noqa: E402


def shifted(mesh, dx, dy):
    kinds, par = mesh
    par = par.copy()
    for k, p in zip(kinds, par):
        p[0] += dx
        p[1] += dy
        if k == 0:
            p[2] += dx
            p[3] += dy
    return kinds, par


CASES = {
    "few_nodes": (lambda: geometry.circle(0.5, 5), 4, (-0.7, -0.6), (0.8, 0.7), 3, 2, 2.0),
    "tile_remainder": (lambda: geometry.polygon(*geometry.star_polygon(7, seed=3), 43), 3, (-1.3, -1.2), (1.2, 1.3),
                       7, 5, 3.0),
    "long_arcs": (lambda: geometry.circle(0.5, 3), 8, (-0.6, -0.6), (0.61, 0.59), 9, 9, 2.0),
    "beyond_the_table": (lambda: geometry.circle(0.5, 12), 8, (-300.0, -280.0), (310.0, 290.0), 5, 4, 4.0),
    "far_from_the_origin": (lambda: shifted(geometry.circle(0.5, 12), 1000.0, -2000.0), 8, (999.3, -2000.6),
                            (1000.6, -1999.4), 7, 7, 3.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("total", [False, True])
def test_field_matches_oracle(name, total):
    make, order, ll, ur, nx, ny, k = CASES[name]
    kinds, par = make()
    so = api.SolutionsOperator(api.BuilderData((kinds, par), order=7), proj=False)
    w = api.wave("Plane", 1.0, angle=0.4)
    tr = api.tp_solve(so, w, k, 1.0, 3.0)
    S, X, Y = api.tp_field_grid(so, w, k, 1.0, 3.0, order, ll, ur, nx, ny, total_field=total, traces=tr)
    ref = O.field_points(kinds, par, tr, w, k, 1.0, 3.0, order, list(zip(X.ravel(), Y.ravel())), total).reshape(nx, ny)
    assert np.abs(S - ref).max() <= 1e-8 * np.abs(ref).max()
