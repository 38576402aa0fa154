"""Many pairs of little more than 1,024 rows: they go to the lane groups once the batch has enough of
them, and to the long-pair kernel before; both bit-exact against the oracle, as are batches that mix
the two with pairs that must stay with the long-pair kernel."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)
SC = (1, 3, 5, 2, 2)


def _driver(sc=SC):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    return d


def _pairs(rng, n, rows, cols):
    a, b = [], []
    for i in range(n):
        m, k = int(rng.integers(rows[0], rows[1] + 1)), int(rng.integers(cols[0], cols[1] + 1))
        w, r = BASES[rng.integers(0, 4, k)], BASES[rng.integers(0, 4, m)]
        if i % 3:  # related over what fits
            c = min(m, k)
            r[m - c:] = w[:c]
            r[rng.random(m) < 0.02] = ord("N" if i % 5 == 0 else "G")
        a.append(r.tobytes())
        b.append(w.tobytes())
    return a, b


def _check(a, b, sc=SC, forms=(FORM_PLAIN, FORM_BATCHED)):
    p = Pairs.from_lists(a, b)
    want = oracle.align_batch(p, sc)
    for form in forms:
        got = _driver(sc).align_pairs(p, form)
        bad = np.nonzero((got != want).any(axis=1))[0]
        assert len(bad) == 0, (len(bad), bad[:4], got[bad[0]], want[bad[0]])


@pytest.mark.parametrize("n", [2990, 3001, 4096, 4097, 9000])
def test_either_side_of_the_rule(built, n):
    """Equal extents: the share is the number of pairs, below and above it, on both sides of the
    one-block order's limit."""
    rng = np.random.default_rng(n)
    _check(*_pairs(rng, n, (1025, 1025), (64, 64)), forms=(FORM_PLAIN,) if n == 9000 else (FORM_PLAIN, FORM_BATCHED))


@pytest.mark.parametrize("sc", [SC, (3, 1, 2, 5, 0), (4, 5, 6, 1, 3)])
def test_rows_of_the_bucket(built, sc):
    """Rows at both ends of the bucket, scores whose bound is above the keys (match 3 and 4), and
    longer pairs beside them."""
    rng = np.random.default_rng(sc[0])
    a, b = [], []
    for rows in ((1024, 1026), (1279, 1281), (1030, 1280)):
        x, y = _pairs(rng, 1200, rows, (1, 120))
        a += x
        b += y
    x, y = _pairs(rng, 12, (1030, 3000), (1000, 2500))
    u, v = _pairs(rng, 600, (30, 900), (30, 400))
    _check(a + x + u, b + y + v, sc)


def test_one_long_pair_among_many(built):
    """A pair with a thousand times the cells keeps the batch with the long-pair kernel."""
    rng = np.random.default_rng(9)
    a, b = _pairs(rng, 5000, (1025, 1100), (20, 40))
    x, y = _pairs(rng, 3, (1100, 1200), (30000, 30000))
    _check(a + x, b + y, forms=(FORM_BATCHED,))
