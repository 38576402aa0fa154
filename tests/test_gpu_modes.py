"""The forward engine's modes (step keys, half and integer arithmetic) at the score bounds where
one gives way to the next, and the score2 sweep's masked edges, against the oracle."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, GPUDriver, Pairs
from mhm2_staging_gb300 import driver as D
from oracle import oracle

pytestmark = pytest.mark.gpu
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _pairs(rng, longest, n=10240):
    """Pairs up to `longest` on both sides, the longest identical (their score is the bound),
    the others related, unrelated or a prefix of one another."""
    a, b = [], []
    for i in range(n):
        if i < 40:
            m = k = longest
        else:
            m, k = (int(x) for x in rng.integers(1, 161 if i % 8 else longest + 1, 2))
            m, k = min(m, longest), min(k, longest)
        w = BASES[rng.integers(0, 4, max(m, k))]
        r = w[:m].copy()
        if i % 3 == 1:
            hit = rng.random(m) < 0.05
            r[hit] = BASES[rng.integers(0, 4, int(hit.sum()))]
            r[rng.random(m) < 0.01] = ord("N")
        elif i % 3 == 2:
            r = BASES[rng.integers(0, 4, m)]
        a.append(r.tobytes())
        b.append(w[:k].tobytes())
    return Pairs.from_lists(a, b)


@pytest.mark.parametrize("longest,sc", [
    (448, (1, 3, 5, 2, 2)), (449, (1, 3, 5, 2, 2)), (96, (2, 4, 4, 2, 1)), (224, (2, 127, 127, 2, 0)),
    (225, (2, 4, 4, 4, 1)), (256, (7, 3, 5, 2, 2)), (257, (7, 3, 5, 2, 2)), (14, (127, 3, 5, 2, 2)),
    (160, (12, 6, 9, 3, 0)), (18, (100, 3, 127, 2, 2)), (192, (1, 0, 7, 7, 0))])
def test_mode_bounds(built, longest, sc):
    torch = pytest.importorskip("torch")
    p = _pairs(np.random.default_rng(longest + sc[0]), longest)
    want = oracle.align_batch(p, sc, score2=True)
    for lane_rows, score2 in ((128, False), (160, False), (160, True)):
        d = GPUDriver()
        d.init(0, 1, sc[0], -sc[1], -sc[2], -sc[3], 0)
        d.set_ambiguity(-sc[4])
        d.set_score2(score2)
        d.fix_batch_config(128, 0, lane_rows, False)
        assert np.array_equal(d.align_pairs(p, FORM_BATCHED), want[:, :5])
        if score2:
            assert np.array_equal(d.last_score2(p.n), want[:, 5:])
    tens = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    dp = D.DevicePairs(*(t.data_ptr() for t in tens), n=p.n, max_a_len=int(p.a_len.max()), max_b_len=int(p.b_len.max()))
    out = torch.full((p.n, 3), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    D.forward_noalloc(dp, out.data_ptr(), (sc[0], -sc[1], -sc[2], -sc[3], -sc[4]))
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want[:, [0, 2, 4]])
