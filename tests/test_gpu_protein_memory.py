"""Device memory of the protein entry point with one very long B among ordinary pairs: only the
int32 kernels' rows follow its length."""
import numpy as np
import pytest

from mhm2_staging_gb300 import GPUDriver, Pairs
from mhm2_staging_gb300.protein import PROTEIN_LETTERS, protein_encoding
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_one_very_long_sequence(built):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    let = np.frombuffer(PROTEIN_LETTERS[:20].encode(), dtype=np.uint8)
    n, cols = 64, 2_000_000
    a = [let[rng.integers(0, 20, 12)].tobytes()] + [let[rng.integers(0, 20, 600)].tobytes() for _ in range(n - 1)]
    b = [let[rng.integers(0, 20, cols)].tobytes()] + [let[rng.integers(0, 20, 500)].tobytes() for _ in range(n - 1)]
    p = Pairs.from_lists(a, b)
    mat = rng.integers(-4, 2, (24, 24)).astype(np.int16)
    np.fill_diagonal(mat, 6)
    d = GPUDriver()
    d.init(0, 1, 1, -1, -11, -1, 0)
    torch.cuda.synchronize()
    small = d.align_protein(p.slice(1, 8), mat, protein_encoding())  # kernels loaded
    free = torch.cuda.mem_get_info()[0]
    got = d.align_protein(p, mat, protein_encoding())
    used = free - torch.cuda.mem_get_info()[0]
    assert np.array_equal(got, oracle.protein_batch(p, mat, protein_encoding(), 11, 1))
    assert np.array_equal(got[1:8], small)
    # H and E of a strip's last row, 8 bytes a column and warp, one warp a pair; an eighth of growth
    # room; sequences and codes twice over; 32 MB for the rest
    assert used < 1.125 * (n * cols * 8 + 4 * (cols + 600 * n)) + (32 << 20), used
