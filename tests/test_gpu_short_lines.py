"""Batches on either side of the lines between the one-launch path and the general one: the route taken
and the results, plain and score2, against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_PLAIN, GPUDriver, Pairs
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)
SC = (1, 3, 5, 2, 2)


def _pairs(rng, n, rows, cols):
    a, b = [], []
    for i in range(n):
        w = BASES[rng.integers(0, 4, cols if i == 0 else int(rng.integers(cols // 8, cols // 4)))]
        m = rows if i == 0 else int(rng.integers(rows // 2, rows + 1))
        at = int(rng.integers(0, max(1, w.shape[0] - m)))
        r = np.resize(w[at:at + m], m) if i % 3 else BASES[rng.integers(0, 4, m)]
        a.append(r.tobytes())
        b.append(w.tobytes())
    return Pairs.from_lists(a, b)


@pytest.mark.parametrize("n,rows,cols,score2,one", [
    (2000, 64, 2000, False, True), (2001, 64, 1500, False, False), (2001, 65, 1500, False, True),
    (2001, 64, 1499, False, True), (1500, 64, 2100, True, True), (1501, 64, 2100, True, False),
    (1501, 64, 1998, True, True), (6500, 256, 1700, False, True), (6501, 256, 1700, False, False),
    (6501, 257, 1700, False, True), (6501, 256, 1692, True, True)])
def test_route_and_results(built, n, rows, cols, score2, one):
    p = _pairs(np.random.default_rng(n + rows + cols), n, rows, cols)
    d = GPUDriver()
    d.init(0, 1, 1, -3, -5, -2, 0)
    d.set_ambiguity(-2)
    d.set_score2(score2)
    want = oracle.align_batch(p, SC, score2=score2)
    assert np.array_equal(d.align_pairs(p, FORM_PLAIN), want[:, :5])
    assert (d.last_timing()["launches"] == 1) == one
    if score2:
        assert np.array_equal(d.last_score2(n), want[:, 5:7])
