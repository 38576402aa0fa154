"""Protein pairs on the keyed int16 kernels and past their limits (rows at the tiles' edges,
strips, scores at the key's capacity, matrices the bytes cannot hold), against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs
from mhm2_staging_gb300.protein import PROTEIN_LETTERS, protein_encoding
from oracle import oracle

pytestmark = pytest.mark.gpu
ENC = protein_encoding()


def _matrix(seed, low, top):
    r = np.random.default_rng(seed)
    m = r.integers(low, 2, (24, 24))
    np.fill_diagonal(m, r.integers(max(1, top - 4), top + 1, 24))
    m[0, 0] = top
    m[1, 2] = low
    return m.astype(np.int16)


def _pairs(seed, rows, cols):
    rng = np.random.default_rng(seed)
    let = np.frombuffer(PROTEIN_LETTERS.encode(), dtype=np.uint8)
    a, b = [], []
    for m in rows:
        for n in cols:
            x, y = let[rng.integers(0, 24, m)], let[rng.integers(0, 24, n)]
            k = min(m, n)
            if (m + n) % 3:
                y[n - k:] = x[:k]
                hit = rng.random(n) < 0.15
                y[hit] = let[rng.integers(0, 24, int(hit.sum()))]
            a.append(x.tobytes())
            b.append(y.tobytes())
    return Pairs.from_lists(a, b)


def _check(p, mat, go, ge):
    d = GPUDriver()
    d.init(0, 1, 1, -1, -go, -ge, 0)
    got = d.align_protein(p, mat, ENC)
    want = oracle.protein_batch(p, mat, ENC, go, ge)
    bad = np.nonzero((got != want).any(axis=1))[0]
    assert len(bad) == 0, (len(bad), bad[:3], got[bad[0]], want[bad[0]])


@pytest.mark.parametrize("low,top,go,ge", [(-4, 9, 11, 1), (-11, 9, 11, 1), (-4, 63, 64, 2), (-1, 5, 1, 1), (0, 1, 3, 5)])
def test_tile_edges(built, low, top, go, ge):
    rows = [1, 2, 64, 127, 128, 129, 191, 192, 193, 255, 256, 257, 383, 384, 385, 511, 512, 513, 1025]
    _check(_pairs(top, rows, [1, 2, 3, 30, 31, 33, 64, 67, 130, 333]), _matrix(top, low, top), go, ge)


@pytest.mark.parametrize("low,top,go,ge", [(-12, 9, 11, 1), (-4, 64, 11, 1), (-4, 63, 65, 1)])
def test_matrices_outside_the_keyed_kernels(built, low, top, go, ge):
    _check(_pairs(3, [1, 128, 300], [5, 129, 300]), _matrix(4, low, top), go, ge)


def test_scores_past_the_keys(built):
    """Near-identical pairs around and past 4032 (and past int16) among ordinary ones."""
    rng = np.random.default_rng(2)
    let = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8)
    a, b = [], []
    for m in (60, 63, 64, 65, 66, 70, 150, 500, 900):
        for _ in range(12):
            x = let[rng.integers(0, 20, m)]
            y = x.copy()
            y[rng.random(m) < 0.01] = ord("A")
            a += [x.tobytes(), x[:40].tobytes()]
            b += [y.tobytes(), y[20:].tobytes()]
    _check(Pairs.from_lists(a, b), _matrix(9, -4, 63), 20, 2)


@pytest.mark.parametrize("n", [1, 4096, 4097])
def test_batch_sizes(built, n):
    rng = np.random.default_rng(n)
    p = _pairs(n, [int(x) for x in rng.integers(1, 300, 64)], [int(x) for x in rng.integers(1, 300, max(1, (n + 63) // 64))])
    p = p.slice(0, n)
    _check(p, _matrix(1, -4, 9), 11, 1)
