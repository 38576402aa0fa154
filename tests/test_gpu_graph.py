"""A captured device batch beside other calls on its handle: replays read and write the handle's
buffers by address, so whatever ran in between must leave them in place or have the graph renewed."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs, workloads
from mhm2_staging_gb300 import serving as S
from oracle import oracle

pytestmark = pytest.mark.gpu
SC = (1, 3, 5, 2, 2)
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _driver(sc=SC):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    return d


def _rows(n, rows, seed):
    """n pairs of `rows` rows (above 512: no short batch), half of them related."""
    rng = np.random.default_rng(seed)
    a, b = [], []
    for i in range(n):
        w = BASES[rng.integers(0, 4, rows + 100)]
        r = w[50:50 + rows].copy() if i % 2 else BASES[rng.integers(0, 4, rows)]
        r[rng.random(rows) < 0.03] = ord("T")
        a.append(r.tobytes())
        b.append(w.tobytes())
    return Pairs.from_lists(a, b)


class _Resident:
    """A batch on the device with its stated extents, and its expected results."""

    def __init__(self, torch, p, sc=SC, score2=False):
        from mhm2_staging_gb300.driver import DevicePairs

        self.torch, self.p = torch, p
        self.keep = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
        self.dp = DevicePairs(*(t.data_ptr() for t in self.keep), p.n, *p.extents())
        self.out = torch.zeros((p.n, 5), dtype=torch.int32, device="cuda")
        self.want = oracle.align_batch(p, sc, score2=score2)

    def run(self, d):
        """Aligns the batch, checks everything it gives, returns the graph replays so far."""
        self.out.fill_(-9)
        self.torch.cuda.synchronize()
        d.align_pairs_device(self.dp, self.out.data_ptr())
        assert np.array_equal(self.out.cpu().numpy(), self.want[:, :5])
        if self.want.shape[1] > 5:
            assert np.array_equal(d.last_score2(self.p.n), self.want[:, 5:7])
        return d.last_timing()["graph_replays"]


@pytest.mark.parametrize("n_short", [40, 5000])
@pytest.mark.parametrize("host", [False, True])
def test_short_score2_batch_in_between(built, n_short, host):
    """Fewer pairs than the captured batch (its count of second-best scores stays its own) and
    more (the shared result arrays are reallocated)."""
    torch = pytest.importorskip("torch")
    big = _Resident(torch, _rows(300, 600, 1), score2=True)
    p = workloads.generate(2, n=n_short, first=7)
    short = _Resident(torch, p, score2=True)
    d = _driver()
    d.set_score2(True)
    launches = []
    for _ in range(3):
        for _ in range(3):
            big.run(d)
            launches.append(d.last_timing()["launches"])
        if host:
            assert np.array_equal(d.align_pairs(p), short.want[:, :5])
            assert np.array_equal(d.last_score2(p.n), short.want[:, 5:7])
        else:
            short.run(d)
        assert d.last_timing()["launches"] == 1
    assert min(launches) > 1 and len(set(launches)) == 1, launches


@pytest.mark.parametrize("late_cigar", [False, True])
@pytest.mark.parametrize("n_block", [300, 3000])
def test_short_block_in_between(built, n_block, late_cigar):
    """Drop-in blocks on the one-launch path, read in place and copied (above 512 KB), with more
    pairs than the captured batch, and with CIGAR mode switched on between their passes."""
    torch = pytest.importorskip("torch")
    big = _Resident(torch, _rows(60, 1100, 2))
    p = workloads.generate(2, n=n_block, first=5)
    want = oracle.align_batch(p, SC)
    reads, ctgs = [p.a(i) for i in range(p.n)], [p.b(i) for i in range(p.n)]
    ma, mb = max(map(len, reads)), max(map(len, ctgs))
    d = _driver()
    replays = []
    for _ in range(3):
        replays.append([big.run(d) for _ in range(3)])
        d.run_kernel_forwards(reads, ctgs, ma, mb)
        d.kernel_block()
        d.set_cigar(late_cigar)
        d.run_kernel_backwards(reads, ctgs, ma, mb)
        d.kernel_block()
        d.set_cigar(False)
        r = d.get_aln_results()
        got = np.stack([r.top_scores32, r.query_begin32, r.query_end32, r.ref_begin32, r.ref_end32], axis=1)
        assert np.array_equal(got, want)
    # every buffer has its size after the first round: the second renews the graph where one
    # moved, the third goes on replaying
    assert replays[2][2] - replays[1][2] == 3, replays


def test_general_calls_in_between(built):
    """A klign call, a block and a host batch on the general path: results stay right, and the
    graph goes on once nothing grows any more."""
    torch = pytest.importorskip("torch")
    from mhm2_staging_gb300.klign import ResidentContigs, generate_candidates, klign_align

    contigs = S.generate_contigs(2 << 20, seed=3)
    resident = ResidentContigs(contigs)
    cand = generate_candidates(contigs, 20000, seed=5)
    big = _Resident(torch, workloads.generate(2, n=9000, first=3))
    host = workloads.generate(1, n=12000, first=9)
    host_want = oracle.align_batch(host, SC)
    reads, ctgs = [host.a(i) for i in range(host.n)], [host.b(i) for i in range(host.n)]
    d = _driver()
    replays, klign = [], []
    for _ in range(4):
        replays.append([big.run(d) for _ in range(3)])
        klign.append(klign_align(d, resident, cand))
        d.run_kernel_forwards(reads, ctgs, 4096, 4096)
        d.run_kernel_backwards(reads, ctgs, 4096, 4096)
        d.kernel_block()
        assert np.array_equal(d.get_aln_results().top_scores32, host_want[:, 0])
    assert all(np.array_equal(klign[0][k], x[k]) for x in klign for k in ("score1", "rstart", "cstop"))
    assert replays[3][2] - replays[2][2] == 3, replays
    # a host batch takes the graph's place, as any other batch of this entry point
    assert np.array_equal(d.align_pairs(host), host_want)
    assert big.run(d) == replays[3][2]
    resident.close()


def test_replayed_cigars_of_large_boxes(built):
    """CIGAR mode, boxes above the register kernels' 512 rows: the generic kernel runs after the
    replay, outside the graph, on the replayed batch's codes."""
    torch = pytest.importorskip("torch")
    sc = (2, 4, 4, 2, 1)
    big = _Resident(torch, _rows(60, 700, 4), sc)
    want, wops, wn = oracle.cigar_batch(big.p, sc, ops_cap=4096)
    d = _driver(sc)
    d.set_cigar(True)
    replays = []
    for _ in range(4):
        replays.append(big.run(d))
        c = d.last_cigar(big.p.n)
        assert np.array_equal(c.nops, wn) and np.array_equal(c.mismatches, want[:, 5])
        assert all(np.array_equal(c.of(i), wops[i, :max(int(wn[i]), 0)]) for i in range(big.p.n))
        assert d.last_timing()["n_cigar_generic"] >= 30
    assert replays == [0, 1, 2, 3], replays
