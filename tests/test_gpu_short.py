"""Short batches (one launch for both passes) and the pair order of larger ones, bit-exact
against the oracle at the sizes where their tiles and bins end."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu
SC = (1, 3, 5, 2, 2)


def _driver(sc=SC):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    return d


def _pairs(rng, rows, cols):
    """One related and one unrelated pair per size, some Ns and lower case among them."""
    bases = np.frombuffer(b"ACGT", dtype=np.uint8)
    a, b = [], []
    for m, n in zip(rows, cols):
        for related in (True, False):
            w = bases[rng.integers(0, 4, n)]
            r = bases[rng.integers(0, 4, m)]
            if related:
                k = min(m, n)
                at = int(rng.integers(0, n - k + 1))
                r[:k] = w[at:at + k]
                hit = rng.random(m) < 0.04
                r[hit] = bases[rng.integers(0, 4, int(hit.sum()))]
                if m > 30:  # one insertion, one deletion
                    r = np.insert(np.delete(r, m // 3), 2 * m // 3, ord("a"))
            r[rng.random(m) < 0.01] = ord("N")
            a.append(r.tobytes())
            b.append(w.tobytes())
    return Pairs.from_lists(a, b)


ROWS = [1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 250, 255, 256]
LONG_ROWS = ROWS + [257, 383, 384, 385, 511, 512]


@pytest.mark.parametrize("rows", [ROWS, LONG_ROWS], ids=["up_to_256", "up_to_512"])
@pytest.mark.parametrize("sc", [SC, (2, 4, 4, 2, 1), (1, 1, 1, 1, 1), (3, 0, 7, 7, 0)])
def test_tile_edges(built, rows, sc):
    rng = np.random.default_rng(len(rows) + sc[1])
    cols = [1, 3, 4, 5, 62, 63, 64, 65, 130, 300, 301, 777, 1024]
    p = _pairs(rng, [m for m in rows for _ in cols], cols * len(rows))
    want = oracle.align_batch(p, sc)
    for form in (FORM_PLAIN, FORM_BATCHED):
        d = _driver(sc)
        assert np.array_equal(d.align_pairs(p, form), want)
        assert d.last_timing()["launches"] == 1
        # the general path on the same pairs
        d.fix_batch_config(128, 0, 160, False)
        assert np.array_equal(d.align_pairs(p, FORM_BATCHED), want)


@pytest.mark.parametrize("sc", [SC, (2, 4, 4, 2, 1), (4, 5, 6, 1, 3)])
def test_second_best_scores(built, sc):
    """Score2 mode at the tiles' and paddings' edges, byte and word path (scores above 255 at
    match 2 and 4), and with CIGAR mode on top."""
    rng = np.random.default_rng(sc[0])
    cols = [1, 7, 8, 9, 15, 16, 17, 64, 120, 121, 128, 129, 300, 305]
    p = _pairs(rng, [m for m in LONG_ROWS for _ in cols], cols * len(LONG_ROWS))
    want = oracle.align_batch(p, sc, score2=True)
    for cigar in (False, True):
        d = _driver(sc)
        d.set_score2(True)
        d.set_cigar(cigar)
        assert np.array_equal(d.align_pairs(p), want[:, :5])
        assert np.array_equal(d.last_score2(p.n), want[:, 5:7])
    wc, _, wn = oracle.cigar_batch(p, sc, ops_cap=2048)
    c = d.last_cigar(p.n)
    assert np.array_equal(c.nops, wn) and np.array_equal(c.mismatches, wc[:, 5])


@pytest.mark.parametrize("n", [1, 31, 1200, 8192, 8193])
def test_batch_sizes(built, n):
    """Host batches read in place and copied, up to and past the largest short batch."""
    p = workloads.generate(1, n=n, first=11)
    want = oracle.align_batch(p, SC)
    d = _driver()
    assert np.array_equal(d.align_pairs(p, FORM_PLAIN), want)
    outs = [d.align_pairs_async(p, FORM_BATCHED) for _ in range(6)]
    d.wait()
    assert all(np.array_equal(o, want) for o in outs)


@pytest.mark.parametrize("n", [4095, 4096, 4097, 20000])
def test_pair_order(built, n):
    """Every pair is aligned once whatever its length class (one-block and two-launch order)."""
    rng = np.random.default_rng(n)
    rows = rng.choice([0, 1, 50, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 256, 257, 300], n)
    cols = rng.choice([0, 1, 3, 4, 100, 103, 104], n)
    cols[:40] = rng.choice([1023, 1024, 1039, 1040, 2047, 2048], 40)
    bases = np.frombuffer(b"ACGT", dtype=np.uint8)
    p = Pairs.from_lists([bases[rng.integers(0, 4, m)].tobytes() for m in rows],
                         [bases[rng.integers(0, 4, k)].tobytes() for k in cols])
    d = _driver()
    d.fix_batch_config(128, 0, 160, False)
    out = np.full((n, 5), -7, dtype=np.int32)
    d.align_pairs(p, FORM_BATCHED, out=out)
    assert np.array_equal(out, oracle.align_batch(p, SC))


def test_protocol_views_and_late_cigar_mode(built):
    """The drop-in calls on a short batch; CIGAR mode switched on between the passes still
    gets its CIGARs."""
    p = workloads.generate(2, n=300, first=5)
    reads, ctgs = [p.a(i) for i in range(p.n)], [p.b(i) for i in range(p.n)]
    ma, mb = max(map(len, reads)), max(map(len, ctgs))
    want = oracle.align_batch(p, SC)
    d = _driver()
    for late in (False, True):
        d.run_kernel_forwards(reads, ctgs, ma, mb)
        d.kernel_block()
        d.set_cigar(late)
        d.run_kernel_backwards(reads, ctgs, ma, mb)
        d.kernel_block()
        r = d.get_aln_results()
        got = np.stack([r.top_scores32, r.query_begin32, r.query_end32, r.ref_begin32, r.ref_end32], axis=1)
        assert np.array_equal(got, want)
        assert np.array_equal(r.top_scores, want[:, 0].astype(np.int16))
    wc, _, wn = oracle.cigar_batch(p, SC, ops_cap=1024)
    c = d.last_cigar(p.n)
    assert np.array_equal(c.nops, wn) and np.array_equal(c.mismatches, wc[:, 5])


def test_device_graph_survives_other_entry_points(built):
    """A captured device batch stays right when another entry point resized the handle's
    buffers in between."""
    torch = pytest.importorskip("torch")
    from mhm2_staging_gb300.driver import DevicePairs

    p, big = workloads.generate(2, n=9000, first=3), workloads.generate(2, n=30000, first=99)
    tens = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    ext = p.extents()
    dp = DevicePairs(*(t.data_ptr() for t in tens), p.n, *ext)
    out = torch.zeros((p.n, 5), dtype=torch.int32, device="cuda")
    d = _driver()
    want = oracle.align_batch(p, SC)
    reads, ctgs = [big.a(i) for i in range(big.n)], [big.b(i) for i in range(big.n)]
    for _ in range(2):
        for _ in range(3):
            out.zero_()
            torch.cuda.synchronize()
            d.align_pairs_device(dp, out.data_ptr())
            assert np.array_equal(out.cpu().numpy(), want)
        d.run_kernel_forwards(reads, ctgs, 2048, 2048)
        d.kernel_block()
