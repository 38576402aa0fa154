"""The allocation-free forward pass on each of its routes (one-launch batches, the ordered keyed
engine, wide pairs among them, the int32 engine), against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import Pairs, workloads
from mhm2_staging_gb300 import driver as D
from oracle import oracle

pytestmark = pytest.mark.gpu


def _run(p, scores, max_a=0, max_b=0):
    torch = pytest.importorskip("torch")
    tens = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    dp = D.DevicePairs(*(t.data_ptr() for t in tens), n=p.n, max_a_len=max_a or int(p.a_len.max()),
                       max_b_len=max_b or int(p.b_len.max()))
    out = torch.full((p.n, 3), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    D.forward_noalloc(dp, out.data_ptr(), tuple([scores[0]] + [-x for x in scores[1:]]))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [1, 200, 8192, 8193, 9728, 9729, 30000])
def test_batch_sizes(built, n):
    p = workloads.generate(1, n=n, first=3)
    assert np.array_equal(_run(p, (1, 3, 5, 2, 2)), oracle.align_batch(p, (1, 3, 5, 2, 2))[:, [0, 2, 4]])


@pytest.mark.parametrize("scores", [(1, 3, 5, 2, 2), (30, 3, 5, 2, 2), (1, 9, 5, 2, 2), (2, 4, 4, 2, 1)])
def test_mixed_lengths_and_scorings(built, scores):
    """Empty sides, strips, pairs whose bound exceeds the int16 keys (match 30), a scoring the
    keyed engine cannot hold (mismatch above gap open), and pairs outside the stated maxima in
    every bucket."""
    parts = [workloads.generate(2, n=11000, first=7), workloads.generate(4, n=30, first=2)]
    a = [q.a(i) for q in parts for i in range(q.n)] + [b"", b"ACGT", b"ACGTTGCA" * 90, b"AC" * 500]
    b = [q.b(i) for q in parts for i in range(q.n)] + [b"ACGT", b"", b"TGCAACGT" * 70, b"CA" * 400]
    p = Pairs.from_lists(a, b)
    want = oracle.align_batch(p, scores)[:, [0, 2, 4]]
    assert np.array_equal(_run(p, scores), want)
    for max_a, max_b in ((100, 3000), (150, 400), (200, 100)):
        cut = want.copy()
        cut[(p.a_len > max_a) | (p.b_len > max_b)] = -1
        assert np.array_equal(_run(p, scores, max_a, max_b), cut)
