"""Begin searches on either side of the rule that gives the widest band classes to a warp each: few and
many of them, in batches of mostly narrow ones and of only wide ones, bit-exact against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _pairs(rng, n, rows, sub, gaps):
    """Reads taken from their windows with substitutions and a deletion and an insertion of up to
    `gaps` bases (the band's width follows from what they leave of the score)."""
    a, b = [], []
    for _ in range(n):
        m = int(rng.integers(rows[0], rows[1] + 1))
        w = BASES[rng.integers(0, 4, m + 150)]
        r = w[60:60 + m].copy()
        hit = rng.random(m) < sub
        r[hit] = BASES[rng.integers(0, 4, int(hit.sum()))]
        g = int(rng.integers(0, gaps + 1))
        if g:
            k = int(rng.integers(m // 3, 2 * m // 3))
            r = np.insert(np.delete(r, slice(k, k + g)), m // 4, BASES[rng.integers(0, 4, g)])
        a.append(r.tobytes())
        b.append(w.tobytes())
    return a, b


@pytest.mark.parametrize("sc", [(1, 3, 5, 2, 2), (2, 4, 4, 2, 1), (1, 1, 1, 1, 1)])
@pytest.mark.parametrize("wide,narrow", [(1, 9000), (300, 9000), (3000, 9000), (9000, 0), (20000, 0)])
def test_wide_searches(built, sc, wide, narrow):
    rng = np.random.default_rng(wide + sc[0])
    a, b = _pairs(rng, wide, (100, 300), 0.15, 12)
    x, y = _pairs(rng, narrow, (80, 150), 0.01, 0)
    order = rng.permutation(wide + narrow)
    a, b = a + x, b + y
    p = Pairs.from_lists([a[i] for i in order], [b[i] for i in order])
    want = oracle.align_batch(p, sc)
    m, mis, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -mis, -go, -ge, 0)
    d.set_ambiguity(-amb)
    for form in (FORM_PLAIN, FORM_BATCHED):
        got = d.align_pairs(p, form)
        bad = np.nonzero((got != want).any(axis=1))[0]
        assert len(bad) == 0, (len(bad), bad[:4], got[bad[0]], want[bad[0]])


def test_rows_past_the_warp_kernel(built):
    """Searches of more rows than a warp holds stay in their class or go to the wavefront kernel."""
    rng = np.random.default_rng(3)
    a, b = _pairs(rng, 1500, (400, 900), 0.1, 40)
    x, y = _pairs(rng, 8000, (60, 200), 0.05, 3)
    p = Pairs.from_lists(a + x, b + y)
    d = GPUDriver()
    d.init(0, 1, 1, -3, -5, -2, 0)
    d.set_ambiguity(-2)
    assert np.array_equal(d.align_pairs(p, FORM_PLAIN), oracle.align_batch(p, (1, 3, 5, 2, 2)))


@pytest.mark.parametrize("n", [8500, 30000])
def test_count_of_wide_searches(built, n):
    """n_rev_wide counts the searches wider than the banded kernels hold (63 cells), not those that a
    rule on the batch gives to other kernels."""
    from test_band_bounds import band_sides

    sc = (1, 3, 5, 2, 2)
    rng = np.random.default_rng(n)
    a, b = _pairs(rng, n, (140, 300), 0.12, 0)
    p = Pairs.from_lists(a, b)
    out = oracle.align_batch(p, sc)
    # searches whose first rows are all their rows: nothing outgrows its band on the way
    keep = [i for i in range(n) if 2 * out[i, 0] + 16 >= out[i, 2] + 1]
    p, out = p.subset(keep), out[keep]
    sides = [band_sides(int(ie) + 1, int(je) + 1, int(s), sc) for s, _, ie, _, je in out]
    want = sum(i + j > 2 * 31 for i, j, _ in sides)
    assert p.n > 8192 * 0.9 and 0 < want < p.n // 2
    d = GPUDriver()
    d.init(0, 1, 1, -3, -5, -2, 0)
    d.set_ambiguity(-2)
    d.fix_batch_config(128, 0, 160, False)  # (not the one-launch path)
    got = d.align_pairs(p, FORM_BATCHED)
    assert np.array_equal(got, out)
    assert d.last_timing()["n_rev_wide"] == want
