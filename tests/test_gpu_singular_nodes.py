"""Coincident and adjacent pairs by the node table (calls of 12 wavenumbers and more)
against the quadrature points themselves (smaller calls): the same sum through 16
interpolation nodes, exact to 5e-17 of the kernel, so T, T', T'' differ by the rounding
of two different orders of summation.  The hypersingular block of T is a difference of
two media's matrices that agree in their leading term, which at small k leaves about a
hundredth of its terms: 1e-16 x 100 x a few, hence 1e-13 (relative Frobenius).  Where a pair is
beyond the table's range (ks D > 8) the points serve it in either call: meshes and
wavenumbers below, above and across that line; the smallest mesh, mixed panels, P0
spaces, orders 2 and 20, and uneven meshes in one launch."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import _capi as C, api, geometry  # noqa: E402

from test_gpu_general_rows import half_disc  # noqa: E402

CASES = {
    "circle": (lambda: geometry.circle(0.25, 24), 9, (0.5, 10.0), 23.4, C.SPACE_P1),
    "lines": (lambda: geometry.polygon(*geometry.star_polygon(9, seed=1), 26), 7, (0.3, 3.0), 5.0, C.SPACE_P1),
    "across_the_limit": (lambda: geometry.polygon(*geometry.star_polygon(9, seed=2), 21), 7, (2.0, 12.0), 9.0,
                         C.SPACE_P1),
    "beyond_the_limit": (lambda: geometry.circle(1.0, 8), 7, (14.0, 20.0), 2.0, C.SPACE_P1),
    "three_panels": (lambda: geometry.circle(0.1, 3), 6, (0.5, 4.0), 3.0, C.SPACE_P1),
    "mixed_panels": (lambda: half_disc(6), 11, (1.0, 6.0), 5.0, C.SPACE_P1),
    "p0": (lambda: geometry.circle(0.25, 11), 8, (1.0, 9.0), 7.0, C.SPACE_P0),
    "order2": (lambda: geometry.circle(0.25, 9), 2, (1.0, 9.0), 7.0, C.SPACE_P1),
    "order20": (lambda: geometry.circle(0.25, 6), 20, (1.0, 9.0), 7.0, C.SPACE_P1),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("d", [0, 1, 2])
def test_nodes_match_the_points(name, d):
    import torch
    make, order, (lo, hi), c_i, space = CASES[name]
    so = api.SolutionsOperator(api.BuilderData(make(), space, space, order=order), proj=False)
    n = 2 * so.data.npanels
    ks = np.linspace(lo, hi, 13)
    T = torch.empty((13, d + 1, n, n), dtype=torch.complex128, device="cuda")
    C.check(C.lib().hbem_gen_sol_op_batch_device(so._h, C.dptr(ks), 13, 1.0, c_i, d, ctypes.c_void_p(T.data_ptr())))
    many = T.cpu().numpy()
    for q in (0, 6, 12):
        C.check(C.lib().hbem_gen_sol_op_batch_device(so._h, C.dptr(ks[q:]), 1, 1.0, c_i, d,
                                                     ctypes.c_void_p(T.data_ptr())))
        one = T[0].cpu().numpy()
        for t in range(d + 1):
            err = np.linalg.norm(many[q, t] - one[t]) / np.linalg.norm(one[t])
            assert err <= 1e-13, (name, ks[q], t, err)


def test_uneven_meshes_in_one_launch():
    meshes = [CASES[m][0]() for m in ("lines", "across_the_limit", "circle")]
    ops = [api.SolutionsOperator(api.BuilderData(m, order=7), proj=False) for m in meshes]
    ks = [np.linspace(0.5, 9.0, 14), np.linspace(2.0, 12.0, 12), np.linspace(0.5, 9.0, 3)]
    many = [t.cpu().numpy() for t in api.gen_sol_op_multi_device(ops, ks, 1.0, [5.0, 9.0, 7.0], d=1)]
    for q in (0, 2):
        one = api.gen_sol_op_multi_device(ops, [k[q:q + 1] for k in ks], 1.0, [5.0, 9.0, 7.0], d=1)
        for a, b in zip(many, one):
            b = b.cpu().numpy()
            for t in range(2):
                assert np.linalg.norm(a[q, t] - b[0, t]) <= 1e-13 * np.linalg.norm(b[0, t])
