"""Protein pairs whose scores leave the int16 kernels' plain keys (4032): swept again with keys above
a base, up to the bound where the int32 kernels take over, in one strip and several, with ties and
bases that move in either half, against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs
from mhm2_staging_gb300.protein import PROTEIN_LETTERS, protein_encoding
from oracle import oracle

pytestmark = pytest.mark.gpu
ENC = protein_encoding()
LET = np.frombuffer(PROTEIN_LETTERS[:20].encode(), dtype=np.uint8)


def _matrix(seed, low, top):
    r = np.random.default_rng(seed)
    m = r.integers(low, 2, (24, 24))
    np.fill_diagonal(m, r.integers(max(1, top - 3), top + 1, 24))
    return m.astype(np.int16)


def _near(rng, n, sub, gaps):
    """A sequence of n residues and a copy with substitutions and a few gaps of up to 40."""
    x = LET[rng.integers(0, 20, n)]
    y = x.copy()
    hit = rng.random(n) < sub
    y[hit] = LET[rng.integers(0, 20, int(hit.sum()))]
    for _ in range(gaps):
        k, g = int(rng.integers(0, y.shape[0])), int(rng.integers(1, 41))
        y = np.delete(y, slice(k, k + g)) if rng.random() < 0.5 else np.insert(y, k, LET[rng.integers(0, 20, g)])
    return x.tobytes(), y.tobytes()


def _check(pairs, mat, go, ge):
    p = Pairs.from_lists([x for x, _ in pairs], [y for _, y in pairs])
    d = GPUDriver()
    d.init(0, 1, 1, -1, -go, -ge, 0)
    got = d.align_protein(p, mat, ENC)
    want = oracle.protein_batch(p, mat, ENC, go, ge)
    bad = np.nonzero((got != want).any(axis=1))[0]
    assert len(bad) == 0, (len(bad), bad[:3], got[bad[0]], want[bad[0]])
    return want


@pytest.mark.parametrize("top,go,ge", [(63, 64, 2), (63, 20, 30), (30, 1, 1), (16, 11, 1), (9, 11, 1)])
def test_rows_and_strips(built, top, go, ge):
    """Every group width and strip count, scores from below the keys' capacity to 29,999 and past it."""
    rng = np.random.default_rng(top + go)
    full = 30000 // top
    rows = sorted({64, 66, 128, 193, 255, 256, 257, 384, 385, 500, 512, 513, 700, 1024, 1025, full - 1, full, full + 1})
    out = []
    for n in rows:
        if n > full + 1:
            continue
        out += [_near(rng, n, 0.0, 0), _near(rng, n, 0.02, 2), _near(rng, n, 0.2, 3)]
        x, y = _near(rng, n, 0.01, 1)
        flank = LET[rng.integers(0, 20, 150)].tobytes()
        out += [(x, flank + y + flank), (flank[:40] + x, y)]
    want = _check(out, _matrix(top, -4, top), go, ge)
    assert (want[:, 0] > 4032).sum() > 10 and (want[:, 0] < 4033).any()


def test_ties_of_high_scores(built):
    """The same high-scoring piece twice in A (the first row wins), in B (the first column wins) and
    in both, at offsets that put the copies in other lanes, halves and strips."""
    rng = np.random.default_rng(8)
    mat = _matrix(3, -4, 20)
    out = []
    for n, gap in ((260, 1), (260, 20), (260, 300), (300, 7), (400, 40)):
        x = LET[rng.integers(0, 20, n)].tobytes()
        s = LET[rng.integers(0, 20, gap)].tobytes()
        out += [(x + s + x, x), (x, x + s + x), (x + s + x, x + s[:1] * gap + x), (s + x + x, x + x + s)]
    want = _check(out, mat, 30, 3)
    assert (want[:, 0] > 4032).all()


@pytest.mark.parametrize("n", [300, 5000])
def test_among_ordinary_pairs(built, n):
    rng = np.random.default_rng(n)
    out = []
    for i in range(n):
        k = int(rng.integers(30, 700))
        out.append(_near(rng, k, 0.01 if i % 7 == 0 else 0.7, 1))
    _check(out, _matrix(5, -4, 11), 11, 1)
