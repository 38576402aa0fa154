"""CIGAR pass, lanes form against the thread form's classes: bands at the widths where a group
size or a class ends, boxes at the row cap, escalations, and a class too large for it."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu
SC = (2, 4, 4, 2, 1)


def _check(p, sc, cap=2048):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    d.set_cigar(True)
    assert np.array_equal(d.align_pairs(p), oracle.align_batch(p, sc))
    want, ops, n = oracle.cigar_batch(p, sc, ops_cap=cap)
    c = d.last_cigar(p.n)
    assert np.array_equal(c.nops, n) and np.array_equal(c.mismatches, want[:, 5])
    assert all(np.array_equal(c.of(i), ops[i, :max(int(n[i]), 0)]) for i in range(p.n))


def _gapped(rng, rows, gaps):
    """Reads cut from a window with the given insertions (+) and deletions (-) spread over it."""
    bases = np.frombuffer(b"ACGT", dtype=np.uint8)
    a, b = [], []
    for n in rows:
        for gap in gaps:
            w = bases[rng.integers(0, 4, n + 40)]
            r = w[20:20 + n].copy()
            r[rng.random(n) < 0.03] = ord("N")
            at = np.linspace(n // 8, n - n // 8, len(gap)).astype(int)[::-1]
            for k, g in zip(at, gap):
                r = np.insert(r, [k] * g, bases[rng.integers(0, 4, g)]) if g > 0 else np.delete(r, slice(k, k - g))
            a.append(r.tobytes())
            b.append(w.tobytes())
    return Pairs.from_lists(a, b)


@pytest.mark.parametrize("sc", [SC, (1, 3, 5, 2, 2), (1, 1, 1, 1, 1), (2, 2, 3, 1, 2)])
def test_band_widths(built, sc):
    rng = np.random.default_rng(sc[1])
    one = [(g,) for k in (1, 2, 3, 4, 6, 7, 8, 9, 14, 15, 16, 17, 31, 32) for g in (k, -k)]
    back = [(k, -k) for k in (1, 2, 3, 4, 7, 8, 9, 16)] + [(1, -2, 3), (-3, 2, 2), (7, -7, 1)]
    _check(_gapped(rng, (60, 129, 250, 400), one + back), sc)


def test_row_cap_and_odd_counts(built):
    rng = np.random.default_rng(5)
    _check(_gapped(rng, (505, 509, 511, 512, 513, 520), [(1,), (-1,), (3,), (-3,), (8,), (-8,), (2, -2)]), SC)
    _check(_gapped(rng, (200,), [(1,)] * 5), SC)  # a warp with idle groups


def test_tie_heavy_and_large_class(built):
    """Low-complexity pairs (many ties), and a class above the lanes form's limit."""
    rng = np.random.default_rng(8)
    bases = np.frombuffer(b"AC", dtype=np.uint8)
    a = [bases[rng.integers(0, 2, int(k))].tobytes() for k in rng.integers(1, 90, 3000)]
    b = [bases[rng.integers(0, 2, int(k))].tobytes() for k in rng.integers(1, 90, 3000)]
    _check(Pairs.from_lists(a, b), SC)
    p = workloads.generate(2, n=130000, first=17)
    d = GPUDriver()
    d.init(0, 1, 2, -4, -4, -2, 0)
    d.set_ambiguity(-1)
    d.set_cigar(True)
    d.align_pairs(p)
    c = d.last_cigar(p.n)
    idx = rng.choice(p.n, 4000, replace=False)
    want, ops, n = oracle.cigar_batch(p.subset(idx), SC, ops_cap=512)
    assert np.array_equal(c.nops[idx], n) and np.array_equal(c.mismatches[idx], want[:, 5])
    assert all(np.array_equal(c.of(int(i)), ops[j, :max(int(n[j]), 0)]) for j, i in enumerate(idx))
