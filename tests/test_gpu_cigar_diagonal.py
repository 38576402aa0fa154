"""CIGARs of boxes on one diagonal, walked sixteen cells at a time: lengths around the vectors,
every alignment of the two sequences to them, mismatches and Ns in the first and last cells."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sc", [(2, 4, 4, 2, 1), (1, 3, 5, 2, 2), (4, 1, 6, 2, 0)])
def test_diagonal_boxes(built, sc):
    rng = np.random.default_rng(sc[0])
    bases = np.frombuffer(b"ACGT", dtype=np.uint8)
    a, b = [], []
    for n in [1, 2, 15, 16, 17, 18, 31, 32, 33, 47, 48, 49, 64, 65, 150, 250, 511, 513]:
        for flips in ((), (3,), (15,), (16,), (14, 15, 16, 17), (n - 4,), tuple(range(5, n - 5, 7))):
            w = bases[rng.integers(0, 4, n + int(rng.integers(0, 9)))]
            at = int(rng.integers(0, len(w) - n + 1))
            r = w[at:at + n].copy()
            for k in flips:
                if 0 <= k < n:
                    r[k] = ord("N") if k % 3 == 0 else bases[(int(np.searchsorted(bases, r[k])) + 1) % 4]
            a.append(r.tobytes())
            b.append(w.tobytes())
    p = Pairs.from_lists(a, b)
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    d.set_cigar(True)
    assert np.array_equal(d.align_pairs(p), oracle.align_batch(p, sc))
    want, ops, n = oracle.cigar_batch(p, sc, ops_cap=1024)
    c = d.last_cigar(p.n)
    assert np.array_equal(c.nops, n) and np.array_equal(c.mismatches, want[:, 5])
    assert all(np.array_equal(c.of(i), ops[i, :max(int(n[i]), 0)]) for i in range(p.n))
