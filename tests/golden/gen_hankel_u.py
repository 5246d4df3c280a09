"""f(u) = H0(sqrt u), g(u) = H1(sqrt u) / sqrt u at the ends, edges and random points of the octaves
that the table of hankel_u.cuh covers, by mpmath with 60 digits: hankel_u_mpmath.json, rows of
[u, Re f, Im f, Re g, Im g] (floats as hexadecimal)."""
import json
import os
import random

import mpmath as mp

HERE = os.path.dirname(os.path.abspath(__file__))
EMIN, EMAX = -110, 18


def points():
    rng = random.Random(20240611)
    for e in range(EMIN, EMAX):
        lo, eps = 2.0 ** e, 2.0 ** -52
        bits = 7 if e < 4 else 8 + (e - 4) // 2
        i = rng.randrange(1, 1 << bits)                       # an interval's lower edge, and just below it
        edge = lo * (1 + i / (1 << bits))
        yield from (lo, edge, edge * (1 - eps / 2) if edge * (1 - eps / 2) < edge else edge - lo * eps, 2 * lo * (1 - eps / 2))
        for _ in range(2 if e < -20 else 4):
            yield lo * (1 + rng.random())
    for n in range(1, 41):                                     # near the zeros of J0 and Y0
        for z in (mp.besseljzero(0, n), mp.besselyzero(0, n)):
            yield float(z * z)


def main():
    mp.mp.dps = 60
    rows = []
    for u in points():
        x = mp.sqrt(mp.mpf(u))
        v = (mp.besselj(0, x), mp.bessely(0, x), mp.besselj(1, x) / x, mp.bessely(1, x) / x)
        rows.append([u.hex()] + [float(t).hex() for t in v])
    with open(os.path.join(HERE, "hankel_u_mpmath.json"), "w") as f:
        json.dump(rows, f, indent=0)


if __name__ == "__main__":
    main()
