"""Long pairs (a block per pair): strips, bands and bases at their edges, bit-exact against the
oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _driver(sc):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    return d


def _mutated(rng, n, sub, indel):
    """A sequence of n bases and a copy with substitutions and indels of up to 30 bases."""
    b = BASES[rng.integers(0, 4, n)]
    a = b.copy()
    hit = rng.random(n) < sub
    a[hit] = BASES[rng.integers(0, 4, int(hit.sum()))]
    for _ in range(int(n * indel)):
        k, g = int(rng.integers(0, a.shape[0])), int(rng.integers(1, 31))
        a = np.insert(a, [k] * g, BASES[rng.integers(0, 4, g)]) if rng.random() < 0.5 else np.delete(a, slice(k, k + g))
    return a.tobytes(), b.tobytes()


def _check(pairs, sc, forms=(FORM_PLAIN, FORM_BATCHED)):
    p = Pairs.from_lists([x for x, _ in pairs], [y for _, y in pairs])
    want = oracle.align_batch(p, sc)
    for form in forms:
        got = _driver(sc).align_pairs(p, form)
        bad = np.nonzero((got != want).any(axis=1))[0]
        assert len(bad) == 0, (len(bad), bad[:4], got[bad[0]], want[bad[0]])


SCORINGS = [(1, 3, 5, 2, 2), (2, 4, 4, 2, 1), (1, 1, 1, 1, 1), (6, 9, 127, 1, 9), (3, 1, 2, 5, 0)]


@pytest.mark.parametrize("sc", SCORINGS)
def test_related_pairs(built, sc):
    rng = np.random.default_rng(sc[0] * 10 + sc[3])
    out = []
    for n in (1025, 1536, 1537, 2048, 2600, 4100):
        for sub, indel in ((0, 0), (0.001, 0.0005), (0.05, 0.002), (0.15, 0.005)):
            a, b = _mutated(rng, n, sub, indel)
            out.append((a, b))
        flank = BASES[rng.integers(0, 4, 700)].tobytes()
        out.append((flank + a, b + flank))
        out.append((a, b[n // 3:]))
        out.append((a[n // 4:] + flank, flank + b))
    _check(out, sc)


def test_extents_and_unrelated(built):
    """B shorter than a lane's skew and than a chunk, low scores in large boxes, Ns, repeats
    (ties across strips), and more pairs than blocks of 16 warps take."""
    rng = np.random.default_rng(4)
    seq = lambda n: BASES[rng.integers(0, 4, n)].tobytes()  # noqa: E731
    out = [(seq(m), seq(n)) for m in (1025, 1100, 3000) for n in (1, 2, 31, 32, 33, 62, 63, 64, 65, 100, 1000, 2500)]
    unit = seq(37)
    out += [(unit * 60, unit * 45), (unit * 30 + seq(900), seq(500) + unit * 30), (b"A" * 1500, b"A" * 1300),
            (b"N" * 1200, seq(1500)), (seq(1300), b"ACGTN" * 400)]
    _check(out, SCORINGS[0])
    _check([(seq(int(m)), seq(int(n))) for m, n in rng.integers(1000, 1400, (320, 2))], SCORINGS[0], (FORM_PLAIN,))


@pytest.mark.parametrize("n,sc", [(9000, (1, 3, 5, 2, 2)), (9000, (3, 4, 5, 2, 2)), (20000, (2, 4, 4, 2, 1))])
def test_high_scores(built, n, sc):
    """Scores past the keys' 4032 and close to (27,000 of 32,000) and past the long kernel's cap."""
    rng = np.random.default_rng(n)
    _check([_mutated(rng, n, 0.001, 0.0002), _mutated(rng, n, 0.02, 0.0005), _mutated(rng, n // 3, 0.3, 0)], sc,
           (FORM_BATCHED,))
