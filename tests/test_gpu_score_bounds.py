"""Scores whose sum lies close to a rounding boundary.  The tensor-core path
sums row maxima in units of 2^-23 and leaves a pair to the ordered sum in
double precision where 100 * sum / rows + 0.5 is within 400 * 2^-24 of a whole
number; just outside of that the fixed-point sum decides.  Digests here are
made so that their exact sums lie inside, just outside and further out, on both
sides of the boundary."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = Fraction(400, 1 << 24)
ELEMS, CUT = 20, 5  # elements of every filter; the cut of a pair of them (CUTOFFS256[4096 // 40])


def overlaps(rng, rows, lo, hi):
    """(bits per filter, common bits) of each row so that the score's distance
    to its boundary, in units of TOL, is in [lo, hi) (negative: below it)."""
    size = 2048 // rows
    while True:
        h = rng.integers(size // 4, size // 2, (1 << 16, rows))
        c = rng.integers(CUT + 1, h + 1)
        x = 100.0 * ((c - CUT) / (h - CUT)).sum(axis=1) / rows + 0.5
        d = (x - np.rint(x)) / float(TOL)
        for k in np.nonzero((d >= lo) & (d < hi))[0]:
            exact = sum(Fraction(int(c[k, r] - CUT), int(h[k, r] - CUT)) for r in range(rows)) * 100 / rows + Fraction(1, 2)
            d_exact = (exact - round(exact)) / TOL
            if lo <= d_exact < hi:
                return h[k], c[k], int(exact // 1)


def pair(g, rng, name, h, c):
    """Digests whose filter r of one side meets only filter r of the other."""
    rows, a, b = len(h), [], []
    for r in range(rows):
        bits = rng.permutation(np.arange(r, 2048 - 2048 % rows, rows))
        common, extra = bits[:c[r]], int(h[r] - c[r])
        for side, own in ((a, bits[c[r]:c[r] + extra]), (b, bits[c[r] + extra:c[r] + 2 * extra])):
            f = np.zeros(2048, dtype=np.uint8)
            f[common] = f[own] = 1
            assert f.sum() == h[r]
            side.append(np.packbits(f, bitorder="little"))
    elems = np.full(rows, ELEMS, dtype=np.uint16)
    return [g.Digest(name + s, 0, rows, 0, 192, 16384, np.concatenate(f), elems) for s, f in (("a", a), ("b", b))]


@pytest.mark.parametrize("rows", [2, 3, 8])
def test_close_to_a_boundary(ctx, oracle, rows):
    import sdhash_gb300 as g

    rng = np.random.default_rng(rows)
    qs, ts, want = [], [], []
    for lo, hi in [(0.05, 0.95), (1.01, 1.5), (1.5, 4), (4, 40)] * 4:
        for a, b in ((lo, hi), (-hi, -lo)):
            h, c, score = overlaps(rng, rows, a, b)
            q, t = pair(g, rng, f"{len(qs):02d}", h, c)
            qs.append(q)
            ts.append(t)
            want.append(score)
    got = ctx.compare_to(ctx.upload(qs), ctx.upload(ts))
    assert list(np.diag(got)) == want
    oq, ot = [oracle.parse(d.to_string()) for d in qs], [oracle.parse(d.to_string()) for d in ts]
    assert np.array_equal(got, oracle.score_cross_matrix(oq, ot))
