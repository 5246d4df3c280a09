"""The Hankel functions of u = x^2 that assembly and fields use at real wavenumbers (hankel_u.cuh),
value by value against mpmath: both sides of octaves' and intervals' edges, random points of every
octave, the zeros of J0 and Y0, both ends of the table and what lies outside it.

Bound per component c of a value of modulus m: rounding of the leading coefficient, the last
multiply-add and the result, 3 x 2^-53 |c|; everything below is at most 2^-7.5 of the modulus, and
the powers from the fourth on, whose sum is taken in FP32, at most 2^-30 with a handful of roundings of
2^-24 -- in all 2^-54 m."""
import json
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300.build import ARCH, CSRC, nvcc  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("hankel_u")
    exe = str(tmp / "probe")
    cmd = [nvcc()] + ARCH + ["-O2", "-std=c++17", os.path.join(HERE, "cpp", "hankel_u_probe.cu"),
                                         os.path.join(CSRC, "hankel_u.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(u):
        np.asarray(u, np.float64).tofile(tmp / "u.bin")
        p = subprocess.run([exe, str(tmp / "u.bin"), str(tmp / "out.bin")], capture_output=True, text=True, timeout=120)
        assert p.returncode == 0, p.stderr
        return np.fromfile(tmp / "out.bin").reshape(-1, 4)
    return run


def test_inside_the_table(evaluate):
    with open(os.path.join(HERE, "golden", "hankel_u_mpmath.json")) as f:
        ref = np.array([[float.fromhex(x) for x in row] for row in json.load(f)])
    got = evaluate(ref[:, 0])
    for c in (0, 2):
        r, g = ref[:, 1 + c:3 + c], got[:, c:c + 2]
        mod = np.hypot(r[:, :1], r[:, 1:])
        bound = 3 * 2.0 ** -53 * np.abs(r) + 2.0 ** -54 * mod
        worst = (np.abs(g - r) / bound).max(axis=1)
        assert worst.max() <= 1, (worst.max(), ref[worst.argmax(), 0])


def test_outside_the_table(evaluate):
    from scipy.special import j0, j1, y0, y1
    u = np.array([2.0 ** 18, 3.7e5, 2.2e11, 2.0 ** -110 * (1 - 2.0 ** -53), 1e-60, 1e-300])
    x = np.sqrt(u)
    got, ref = evaluate(u), np.stack([j0(x), y0(x), j1(x) / x, y1(x) / x], 1)
    for c in (0, 2):   # both reduce the argument: some roundings of x itself
        mod = np.hypot(ref[:, c], ref[:, c + 1])
        assert (np.abs(got[:, c:c + 2] - ref[:, c:c + 2]).max(axis=1) <= 8 * 2.2e-16 * (1 + x) * mod).all()
    # coincidence of the two points, and not a number
    assert np.array_equal(evaluate([0.0, -1.0]), [[1, 0, 0, 0], [1, 0, 0, 0]])
    assert np.isnan(evaluate([np.nan])).all()
