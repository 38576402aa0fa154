"""Plain batches of few pairs on the general path: one bucket for all of them, on 8 or 16 lanes by the
longest A and the pairs, at both sides of every line, against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_PLAIN, GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _pairs(rng, n, longest, cols):
    a, b = [], []
    for i in range(n):
        m = longest if i < 3 else int(rng.integers(0, longest + 1))
        k = cols if i < 2 else int(rng.integers(0, 120))
        w = BASES[rng.integers(0, 4, k)]
        r = BASES[rng.integers(0, 4, m)]
        if i % 3:
            c = min(m, k)
            r[:c] = w[:c]
            r[rng.random(m) < 0.03] = ord("A")
        a.append(r.tobytes())
        b.append(w.tobytes())
    return Pairs.from_lists(a, b)


@pytest.mark.parametrize("longest", [1, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 256, 257, 600])
@pytest.mark.parametrize("n", [5, 1300, 3700, 6200, 9728, 9729])
def test_one_bucket(built, longest, n):
    """(B of 8,300 columns, or more pairs than a short batch, keeps the batch on the general path.)"""
    p = _pairs(np.random.default_rng(longest * 7 + n), n, longest, 8300)
    d = GPUDriver()
    d.init(0, 1, 1, -3, -5, -2, 0)
    d.set_ambiguity(-2)
    got = d.align_pairs(p, FORM_PLAIN)
    assert d.last_timing()["launches"] > 1
    want = oracle.align_batch(p, (1, 3, 5, 2, 2))
    bad = np.nonzero((got != want).any(axis=1))[0]
    assert len(bad) == 0, (len(bad), bad[:4], got[bad[0]], want[bad[0]])


@pytest.mark.parametrize("sc", [(2, 4, 4, 2, 1), (14, 3, 5, 2, 2), (30, 9, 20, 3, 2)])
@pytest.mark.parametrize("longest", [100, 160, 250])
def test_bounds_above_the_keys(built, sc, longest):
    """Scores up to and past the keys of a bucket wider than a pair's own rows need, score2 mode too."""
    p = _pairs(np.random.default_rng(longest + sc[0]), 2500, longest, 8300)
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    want = oracle.align_batch(p, sc, score2=True)
    assert np.array_equal(d.align_pairs(p, FORM_PLAIN), want[:, :5])
    d.set_score2(True)
    assert np.array_equal(d.align_pairs(p, FORM_PLAIN), want[:, :5])
    assert np.array_equal(d.last_score2(p.n), want[:, 5:7])
