"""The allocation-free forward pass after its set-up call: every later route only launches, so it can be
captured into a CUDA graph, and takes no device memory."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

# A process of its own: kernels are loaded when first used, so what an earlier test used is loaded here.
SCRIPT = r'''
import numpy as np
import torch
from mhm2_staging_gb300 import Pairs, workloads
from mhm2_staging_gb300 import driver as D
from oracle import oracle

rng = np.random.default_rng(1)
base = np.frombuffer(b"ACGT", dtype=np.uint8)

def batch(n, rows, cols):
    w = [base[rng.integers(0, 4, cols)] for _ in range(n)]
    return Pairs.from_lists([x[20:20 + rows].tobytes() for x in w], [x.tobytes() for x in w])

def upload(p):
    t = [torch.from_numpy(x).cuda() for x in (p.a_seq, p.a_off, p.a_len, p.b_seq, p.b_off, p.b_len)]
    return t, D.DevicePairs(*(x.data_ptr() for x in t), n=p.n, max_a_len=int(p.a_len.max()), max_b_len=int(p.b_len.max()))

first = upload(workloads.generate(1, n=9000, first=3))
# one-launch batches of every kernel: up to 256 rows and above, scores up to 448 and above
todo = [(batch(50, 150, 300), (1, 3, 5, 2, 2)), (batch(50, 150, 300), (4, 3, 5, 2, 2)),
        (batch(20, 400, 700), (1, 3, 5, 2, 2)), (batch(20, 400, 700), (3, 3, 5, 2, 2))]
dev = [upload(p) for p, _ in todo]
outs = [torch.full((p.n, 3), -7, dtype=torch.int32, device="cuda") for p, _ in todo]
out = torch.zeros((9000, 3), dtype=torch.int32, device="cuda")
stream = torch.cuda.Stream()
D.forward_noalloc(first[1], out.data_ptr(), stream=stream.cuda_stream)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    pass
free = torch.cuda.mem_get_info()[0]
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    for (p, sc), (_, dp), o in zip(todo, dev, outs):
        D.forward_noalloc(dp, o.data_ptr(), (sc[0], *(-x for x in sc[1:])), stream=stream.cuda_stream)
used = free - torch.cuda.mem_get_info()[0]
graph.replay()
torch.cuda.synchronize()
for (p, sc), o in zip(todo, outs):
    assert np.array_equal(o.cpu().numpy(), oracle.align_batch(p, sc)[:, [0, 2, 4]])
print("captured, bytes taken:", used)
'''


def test_short_batches_captured_after_a_long_first_call(built):
    pytest.importorskip("torch")
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, CUDA_MODULE_LOADING="LAZY", PYTHONPATH=str(root))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "captured" in r.stdout
    print(r.stdout)
