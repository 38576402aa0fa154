"""Batches of empty sequences only, on the general path: every pair gets SSW's empty result and
nothing of the batch before it."""
import numpy as np
import pytest

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sc", [(2, 4, 2, 5, 1), (1, 3, 5, 2, 2)])  # (gap open below gap extend: no short batch)
@pytest.mark.parametrize("side", ["a", "b", "both"])
@pytest.mark.parametrize("n", [1, 40, 8193, 9729])
def test_all_empty(built, sc, side, n):
    m, x, go, ge, amb = sc
    d = GPUDriver()
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    before = workloads.generate(2, n=10000, first=1)
    want = oracle.align_batch(before, sc)
    p = Pairs.from_lists([b"" if side != "b" else b"ACGT" * 20] * n, [b"" if side != "a" else b"ACGTT" * 30] * n)
    for form in (FORM_PLAIN, FORM_BATCHED):
        assert np.array_equal(d.align_pairs(before, form), want)
        out = np.full((n, 5), -7, dtype=np.int32)
        d.align_pairs(p, form, out=out)
        assert np.array_equal(out, np.tile(np.array([0, -1, -1, 0, 0], np.int32), (n, 1)))
        reads, ctgs = [p.a(i) for i in range(n)], [p.b(i) for i in range(n)]
        d.set_form(form)
        d.run_kernel_forwards(reads, ctgs, 200, 200)
        d.run_kernel_backwards(reads, ctgs, 200, 200)
        d.kernel_block()
        r = d.get_aln_results()
        assert (r.top_scores32 == 0).all() and (r.query_begin32 == -1).all() and (r.query_end32 == -1).all()
