"""Pairs a batch could not align end its call in an error, through every entry point that can meet
them: waits between the blocks of long pairs that give up (a limit of no polls: the kernels go on
without waiting and return)."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs
from mhm2_staging_gb300.serving import Contigs
from oracle import oracle

pytestmark = pytest.mark.gpu
SC = (1, 3, 5, 2, 2)
BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _driver():
    d = GPUDriver()
    d.init(0, 1, 1, -3, -5, -2, 0)
    d.set_ambiguity(-2)
    return d


def _batch(seed):
    """A few pairs of 1.3-3 kb among short ones, all related."""
    rng = np.random.default_rng(seed)
    a, b = [], []
    for n in (100, 1300, 250, 2000, 3000, 150):
        w = BASES[rng.integers(0, 4, n + 60)]
        r = w[30:30 + n].copy()
        r[rng.random(n) < 0.01] = ord("A")
        a.append(r.tobytes())
        b.append(w.tobytes())
    return Pairs.from_lists(a, b)


def test_batch_calls(built):
    p = _batch(1)
    want = oracle.align_batch(p, SC)
    d = _driver()
    for form in (FORM_PLAIN, FORM_BATCHED):
        d.set_wait_limit(0)
        with pytest.raises(RuntimeError, match="status 7.*pairs were not aligned"):
            d.align_pairs(p, form)
        d.align_pairs_async(p, form)
        with pytest.raises(RuntimeError, match="status 7"):
            d.wait()
        d.set_wait_limit()
        assert np.array_equal(d.align_pairs(p, form), want)


def test_captured_batch(built):
    torch = pytest.importorskip("torch")
    from mhm2_staging_gb300.driver import DevicePairs

    p = _batch(2)
    keep = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    dp = DevicePairs(*(t.data_ptr() for t in keep), p.n, *p.extents())
    out = torch.zeros((p.n, 5), dtype=torch.int32, device="cuda")
    d = _driver()
    d.set_wait_limit(0)
    for _ in range(3):  # run, captured, replayed
        with pytest.raises(RuntimeError, match="status 7"):
            d.align_pairs_device(dp, out.data_ptr())
    d.set_wait_limit()
    for _ in range(3):
        d.align_pairs_device(dp, out.data_ptr())
        assert np.array_equal(out.cpu().numpy(), oracle.align_batch(p, SC))


def test_drop_in_calls_by_pass(built):
    """The forward pass's waits, and the begin pass's alone."""
    p = _batch(3)
    want = oracle.align_batch(p, SC)
    reads, ctgs = [p.a(i) for i in range(p.n)], [p.b(i) for i in range(p.n)]
    d = _driver()
    for forward, begin in ((0, 0), (1 << 22, 0), (1 << 22, 1 << 22)):
        d.set_wait_limit(forward)
        d.run_kernel_forwards(reads, ctgs, 4096, 4096)
        if forward == 0:
            with pytest.raises(RuntimeError, match="status 7"):
                d.kernel_block()
        else:
            d.kernel_block()
            assert np.array_equal(d.get_aln_results().query_end32, want[:, 2])
        d.set_wait_limit(begin)
        d.run_kernel_backwards(reads, ctgs, 4096, 4096)
        if begin == 0:
            with pytest.raises(RuntimeError, match="status 7"):
                d.kernel_block()
        else:
            d.kernel_block()
            assert np.array_equal(d.get_aln_results().query_begin32, want[:, 1])


def test_klign_call(built):
    """Candidates whose reads are long pairs."""
    from mhm2_staging_gb300.klign import Candidates, ResidentContigs, klign_align

    rng = np.random.default_rng(4)
    ctg = BASES[rng.integers(0, 4, 6000)].copy()
    n, size, kmer = 4, 2500, 31
    at = np.array([0, 700, 1900, 3500])
    reads = np.stack([ctg[x:x + size] for x in at])
    reads[:, 40::97] = ord("C")
    cand = Candidates(reads.reshape(-1).copy(), np.arange(n, dtype=np.int64) * size, np.full(n, size, np.int32),
                      np.zeros(n, np.int32), at.astype(np.int32), np.zeros(n, np.int32), np.zeros(n, np.uint8), kmer)
    resident = ResidentContigs(Contigs(ctg, np.zeros(1, np.int64), np.array([6000], np.int32)))
    d = _driver()
    d.set_wait_limit(0)
    with pytest.raises(RuntimeError, match="status 7"):
        klign_align(d, resident, cand)
    d.set_wait_limit()
    got = klign_align(d, resident, cand)
    assert got["n_aligned"] == n and (got["score1"] > 2000).all()
    resident.close()


def test_pair_beyond_the_stated_extents(built):
    """A long pair whose B is longer than the batch's stated longest B: the kernels' scratch ends
    there."""
    torch = pytest.importorskip("torch")
    from mhm2_staging_gb300.driver import DevicePairs

    rng = np.random.default_rng(5)
    w = BASES[rng.integers(0, 4, 4000)]
    p = Pairs.from_lists([w[100:1700].tobytes(), w[500:3500].tobytes()], [w[:2000].tobytes(), w.tobytes()])
    keep = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    ma, mb, cells, ab, bb = p.extents()
    out = torch.zeros((p.n, 5), dtype=torch.int32, device="cuda")
    d = _driver()
    with pytest.raises(RuntimeError, match="status 7.*1 pairs were not aligned"):
        d.align_pairs_device(DevicePairs(*(t.data_ptr() for t in keep), p.n, ma, 2000, cells, ab, bb), out.data_ptr())
    want = oracle.align_batch(p, SC)
    assert np.array_equal(out.cpu().numpy()[0], want[0])
    d.align_pairs_device(DevicePairs(*(t.data_ptr() for t in keep), p.n, ma, mb, cells, ab, bb), out.data_ptr())
    assert np.array_equal(out.cpu().numpy(), want)


def test_limits_of_the_knob(built):
    d = _driver()
    for bad in (-1, (1 << 22) + 1):
        with pytest.raises(RuntimeError, match="status 2"):
            d.set_wait_limit(bad)
