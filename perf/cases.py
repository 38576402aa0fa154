"""Measured cases of the alignment library: what its users call, over the sizes they call it with.

A case is a batch of (A, B) sequence pairs -- A the read (the rows), B the contig window
(the columns) -- through one public entry point:

  host      GPUDriver.align_pairs on host arrays (copies in and results out are part of it)
  device    GPUDriver.align_pairs_device on a resident batch, optionally in score2 or CIGAR mode
  block     klign's drop-in sequence: forwards, block, backwards, block, results
  klign     klign_align: seed-hit candidates against resident contigs
  serving   one request batch through Server.submit / Server.wait
  protein   GPUDriver.align_protein
  noalloc   forward_noalloc

Pair mixes (sizes of the repository's own workloads): "fixed" 150 bp reads in 300 bp
windows; "mix" reads of 100-250 bp in windows 50-774 bases longer, 30% of them unrelated;
"uneven" 60% 150 bp, 30% 250 bp and 10% trimmed reads against lognormal windows; "longref"
250 bp reads against 2-8 kb; "longpair" both sides of 1-12 kb (long reads or contigs).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mhm2_staging_gb300 import FORM_BATCHED, FORM_PLAIN, GPUDriver, Pairs
from mhm2_staging_gb300.driver import DevicePairs, forward_noalloc
from mhm2_staging_gb300.klign import Candidates, ResidentContigs, klign_align
from mhm2_staging_gb300.protein import PROTEIN_LETTERS, protein_encoding
from mhm2_staging_gb300.serving import Contigs, Requests, Server

DEV = "cuda"
FORMS = {"plain": FORM_PLAIN, "batched": FORM_BATCHED}
KLIGN = (1, 3, 5, 2, 2)      # match, mismatch, gap open, gap extend, ambiguity of klign's rounds
ASSEMBLY = (2, 4, 4, 2, 1)   # klign's post-assembly alignment, which asks for CIGARs
FLANK = 200                  # serving windows: read +- 200 bases
KMER = 31


def listed():
    return [
        # a rank's last few candidates: one short call, all latency
        {"name": "host_tiny", "kind": "host", "mix": "fixed", "n": 32, "form": "plain"},
        # klign's block of 20,000 pairs in its own call sequence (the default form)
        {"name": "block_20k", "kind": "block", "mix": "mix", "n": 20000, "form": "plain"},
        # a host program that collects large batches and hands them over at once
        {"name": "host_mix", "kind": "host", "mix": "mix", "n": 150001, "form": "batched"},
        # the main path at throughput: a resident batch of uneven reads and windows
        {"name": "device_uneven", "kind": "device", "mix": "uneven", "n": 800000, "form": "batched", "mode": "plain"},
        # reads against long references
        {"name": "device_longref", "kind": "device", "mix": "longref", "n": 30011, "form": "batched", "mode": "plain"},
        # few long pairs: long reads or contigs against contigs, near-identical ones among them
        {"name": "device_longpair", "kind": "device", "mix": "longpair", "n": 60, "form": "batched", "mode": "plain"},
        # klign's CPU path keeps the second-best score
        {"name": "device_score2", "kind": "device", "mix": "uneven", "n": 100000, "form": "batched", "mode": "score2"},
        # the post-assembly alignment writes SAM records: CIGARs and mismatches
        {"name": "device_cigar", "kind": "device", "mix": "uneven", "n": 100000, "form": "batched", "mode": "cigar"},
        # klign's caller side: candidates of one round against the resident contigs
        {"name": "klign_100k", "kind": "klign", "n": 100000, "form": "batched", "mode": "plain"},
        # one request batch of a serving loop at low load
        {"name": "serving_4k", "kind": "serving", "n": 4000, "form": "batched"},
        # translated reads against a protein set
        {"name": "protein_20k", "kind": "protein", "n": 20000, "lo": 100, "hi": 500},
        # a pipeline that hands the library no memory
        {"name": "noalloc_50k", "kind": "noalloc", "mix": "mix", "n": 50000},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["host", "block", "device", "device", "device", "klign", "serving", "protein", "noalloc"])
    form = rng.choice(["plain", "batched"])
    if kind == "host":
        return {"kind": kind, "mix": rng.choice(["fixed", "mix", "uneven"]), "n": log(1, 150000), "form": form}
    if kind == "block":
        return {"kind": kind, "mix": rng.choice(["fixed", "mix", "uneven"]), "n": log(16, 20000), "form": form}
    if kind == "device":
        mode = rng.choice(["plain", "score2", "cigar"])
        mix = rng.choice(["fixed", "mix", "uneven", "longref", "longpair"]) if mode == "plain" else "uneven"
        top = {"longref": 20000, "longpair": 60}.get(mix, 100000)
        return {"kind": kind, "mix": mix, "n": log(4, top), "form": form if mix != "longpair" else "batched",
                "mode": mode}
    if kind == "klign":
        return {"kind": kind, "n": log(64, 100000), "form": form, "mode": rng.choice(["plain", "score2"])}
    if kind == "serving":
        return {"kind": kind, "n": log(64, 32000), "form": "batched"}
    if kind == "protein":
        lo = log(20, 200)
        return {"kind": kind, "n": log(16, 20000), "lo": lo, "hi": log(lo + 1, 500)}
    return {"kind": kind, "mix": rng.choice(["fixed", "mix", "uneven"]), "n": log(16, 50000)}


# ---- inputs (made on the device from the seed) ---------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uni(g, lo, hi, n):  # integers in [lo, hi]
    return torch.randint(int(lo), int(hi) + 1, (n,), generator=g, device=DEV)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV)


def _bases(g, shape, letters=b"ACGT"):
    k = torch.frombuffer(bytearray(letters), dtype=torch.uint8).to(DEV)
    return k[torch.randint(0, len(letters), shape, generator=g, device=DEV)]


def _offsets(lens):
    off = torch.zeros_like(lens)
    off[1:] = torch.cumsum(lens, 0)[:-1]
    return off


def _copies(g, arena, start, lens, span, sub, indel, n_rate, fresh, letters=b"ACGT"):
    """Reads copied from the arena at `start` (up to `span` bases of it) with substitutions,
    insertions, deletions and Ns at the given rates; fresh reads are random."""
    n, width = lens.shape[0], int(lens.max())
    step = max(1, (64 << 20) // width)
    out = []
    for i in range(0, n, step):
        s = slice(i, min(i + step, n))
        k = s.stop - s.start
        t = torch.arange(width, device=DEV)
        gap = _rand(g, k, width)
        ins = gap < indel[s, None] / 2
        dele = (gap >= indel[s, None] / 2) & (gap < indel[s, None])
        adv = (1 + dele.int() - ins.int())
        src = torch.cumsum(adv, 1, dtype=torch.int32) - adv
        over = src >= span[s, None]
        src = torch.minimum(src.long(), (span[s, None] - 1).clamp(min=0))
        base = arena[start[s, None] + src]
        swap = ins | over | fresh[s, None] | (_rand(g, k, width) < sub[s, None])
        base = torch.where(swap, _bases(g, (k, width), letters), base)
        if n_rate > 0:
            base = torch.where(_rand(g, k, width) < n_rate, torch.full_like(base, ord("N")), base)
        out.append(base[t[None, :] < lens[s, None]])
    return torch.cat(out)


def _pairs(mix, n, g):
    """(a, a_off, a_len, b, b_off, b_len) of a mix, on the device."""
    fresh = torch.zeros(n, dtype=torch.bool, device=DEV)
    n_rate = 0.0
    if mix == "fixed":
        la, lb = torch.full((n,), 150, device=DEV), torch.full((n,), 300, device=DEV)
        sub, indel = torch.full((n,), 0.02, device=DEV), torch.full((n,), 0.005, device=DEV)
    elif mix == "mix":
        la = _uni(g, 100, 250, n)
        lb = (la + _uni(g, 50, 774, n)).clamp(max=1024)
        sub, indel = torch.full((n,), 0.02, device=DEV), torch.full((n,), 0.005, device=DEV)
        fresh, n_rate = _rand(g, n) < 0.3, 0.001
    elif mix == "uneven":
        u = _rand(g, n)
        la = torch.where(u < 0.6, 150, torch.where(u < 0.9, 250, _uni(g, 50, 150, n)))
        lb = torch.exp(math.log(400) + 0.6 * torch.randn(n, generator=g, device=DEV)).long().clamp(64, 2048)
        sub, indel = 0.01 + 0.03 * _rand(g, n), 0.002 + 0.008 * _rand(g, n)
    elif mix == "longref":
        la, lb = torch.full((n,), 250, device=DEV), _uni(g, 2048, 8192, n)
        close = _rand(g, n) < 0.2
        sub, indel = torch.where(close, 0.001, 0.02), torch.where(close, 0.0, 0.005)
    else:  # longpair
        la = torch.exp(math.log(1000) + math.log(12) * _rand(g, n)).long()
        lb = (la.float() * (0.8 + 0.4 * _rand(g, n))).long().clamp(1000, 12000)
        close = _rand(g, n) < 0.3
        sub, indel = torch.where(close, 0.001, 0.05), torch.where(close, 0.0002, 0.02)
    la, lb = la.long(), lb.long()
    b_off = _offsets(lb)
    b = _bases(g, (int(lb.sum()),))
    room = (lb - la).clamp(min=0)
    pos = (_rand(g, n) * (room + 1)).long().clamp(max=room)
    a = _copies(g, b, b_off + pos, la, lb - pos, sub, indel, n_rate, fresh)
    return a, _offsets(la), la, b, b_off, lb


def _device_pairs(p):
    a, ao, al, b, bo, bl = p
    al, bl = al.int(), bl.int()
    keep = (a, ao, al, b, bo, bl)
    cells = float((al.double() * bl.double()).sum())
    return keep, DevicePairs(*(t.data_ptr() for t in keep), al.shape[0], int(al.max()), int(bl.max()), cells,
                             a.shape[0], b.shape[0])


def _host_pairs(p, pinned):
    a, ao, al, b, bo, bl = p
    host = []
    for t in (a, ao, al.int(), b, bo, bl.int()):
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
        h.copy_(t)
        host.append(h.numpy())
    return Pairs(*host)


def _protein_matrix():
    """A 24 x 24 matrix of the usual shape: 4..9 on the diagonal, -4..3 off it, unknowns at -1."""
    r = np.random.default_rng(24)
    m = r.integers(-4, 2, (24, 24))
    m = np.minimum(m, m.T)
    close = r.random((24, 24)) < 0.04
    m[close & close.T] = 2
    np.fill_diagonal(m, r.integers(4, 10, 24))
    m[22, :] = m[:, 22] = -1
    m[23, :] = m[:, 23] = -4
    m[23, 23] = 1
    return m.astype(np.int16)


def _contigs(g, total):
    """Contigs of lognormal length (median 2 kb) on the device: arena, offsets, lengths."""
    n = max(8, total // 3300)
    ln = torch.exp(math.log(2000) + torch.randn(n, generator=g, device=DEV)).long().clamp(300, 200000)
    return _bases(g, (int(ln.sum()),)), _offsets(ln), ln


def _placed_reads(g, contigs, n, exact_frac, sub, indel):
    arena, off, ln = contigs
    cid = _uni(g, 0, ln.shape[0] - 1, n)
    la = _uni(g, 100, 250, n)
    pos = (_rand(g, n) * (ln[cid] - la + 1)).long().clamp(max=ln[cid] - la)
    mut = (_rand(g, n) >= exact_frac).float()
    return cid, la, pos, mut * sub, mut * indel


_COMP = np.full(256, ord("N"), dtype=np.uint8)
for _x, _y in zip(b"ACGTN", b"TGCAN"):
    _COMP[_x] = _y


def _candidates(g, contigs, n):
    arena, off, ln = contigs
    cid, la, pos, sub, indel = _placed_reads(g, contigs, n, 0.4, 0.02, 0.002)
    reads = _copies(g, arena, off[cid] + pos, la, ln[cid] - pos, sub, indel, 0.0005,
                    torch.zeros(n, dtype=torch.bool, device=DEV))
    seed = (_rand(g, n) * (la - KMER + 1)).long().clamp(max=la - KMER)
    pic = torch.minimum(pos + seed, ln[cid] - KMER)
    minus = _rand(g, n) < 0.5
    rc = _rand(g, n) < 0.5
    ro = _offsets(la)
    # reads found on the other strand are the reverse complements
    own = torch.repeat_interleave(torch.arange(n, device=DEV), la)
    at = torch.arange(reads.shape[0], device=DEV) - ro[own]
    flip = reads[ro[own] + la[own] - 1 - at]
    comp = torch.from_numpy(_COMP).to(DEV)[flip.long()]
    reads = torch.where(minus[own], comp, reads)
    pir = torch.where(minus, la - KMER - seed, seed)
    strand = rc.int() | ((rc ^ minus).int() << 1)

    def host(t, dt):
        return t.to(dt).cpu().numpy()

    return Candidates(host(reads, torch.uint8), host(ro, torch.int64), host(la, torch.int32),
                      host(cid, torch.int32), host(pic, torch.int32), host(pir, torch.int32),
                      host(strand, torch.uint8), KMER)


def _requests(g, contigs, n):
    arena, off, ln = contigs
    cid, la, pos, sub, indel = _placed_reads(g, contigs, n, 0.0, 0.02, 0.0)
    reads = _copies(g, arena, off[cid] + pos, la, ln[cid] - pos, sub, indel, 0.0,
                    torch.zeros(n, dtype=torch.bool, device=DEV))
    return Requests(reads.cpu().numpy(), _offsets(la).cpu().numpy(), la.int().cpu().numpy(),
                    cid.int().cpu().numpy(), pos.int().cpu().numpy())


def _protein_pairs(case, g):
    n = case["n"]
    letters = PROTEIN_LETTERS[:20].encode()
    la, lb = _uni(g, case["lo"], case["hi"], n), _uni(g, case["lo"], case["hi"], n)
    bo = _offsets(lb)
    b = _bases(g, (int(lb.sum()),), letters)
    sub, indel = 0.1 + 0.5 * _rand(g, n), torch.full((n,), 0.02, device=DEV)
    a = _copies(g, b, bo, la, lb, sub, indel, 0.0, _rand(g, n) < 0.3, letters)
    return a, _offsets(la), la, b, bo, lb


def _contig_bytes(case):
    return 16 << 20 if case["n"] > 2000 else 2 << 20


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "klign":
        contigs = _contigs(g, _contig_bytes(case))
        return contigs, _candidates(g, contigs, case["n"])
    if kind == "serving":
        contigs = _contigs(g, _contig_bytes(case))
        return contigs, _requests(g, contigs, case["n"])
    if kind == "protein":
        return _protein_pairs(case, g)
    return _pairs(case["mix"], case["n"], g)


def _scores(case):
    return ASSEMBLY if case.get("mode") == "cigar" else KLIGN


def _driver(case):
    d = GPUDriver()
    m, x, go, ge, amb = (11, 3, 11, 1, 2) if case["kind"] == "protein" else _scores(case)
    d.init(0, 1, m, -x, -go, -ge, 0)
    d.set_ambiguity(-amb)
    d.set_form(FORMS[case.get("form", "plain")])
    d.set_score2(case.get("mode") == "score2")
    d.set_cigar(case.get("mode") == "cigar")
    return d


def prepare(case, seed):
    kind = case["kind"]
    made = _inputs(case, seed)
    st = {"kind": kind, "form": FORMS[case.get("form", "plain")], "mode": case.get("mode", "plain"), "n": case["n"]}
    if kind == "noalloc":
        st["keep"], st["dev"] = _device_pairs(made)
        st["out"] = torch.zeros((case["n"], 3), dtype=torch.int32, device=DEV)
    elif kind == "serving":
        (arena, off, ln), st["req"] = made
        st["srv"] = Server(hbm_budget=4 << 30)
        st["srv"].load_contigs(Contigs(arena.cpu().numpy(), off.cpu().numpy(), ln.int().cpu().numpy()))
    else:
        st["drv"] = _driver(case)
        if kind == "device":
            st["keep"], st["dev"] = _device_pairs(made)
            n = case["n"]
            st["out"] = torch.zeros((n, 5), dtype=torch.int32, device=DEV)
            if st["mode"] == "cigar":  # about 15 ops a pair come back; unused entries stay 0
                st["cigars"] = [np.zeros(k, dtype=t) for k, t in ((n, np.int32), (n, np.int32), (n + 1, np.int64),
                                                                  (40 * n, np.uint32))]
        elif kind == "klign":
            (arena, off, ln), st["cand"] = made
            st["contigs"] = ResidentContigs(Contigs(arena.cpu().numpy(), off.cpu().numpy(), ln.int().cpu().numpy()))
        elif kind == "protein":
            st["pairs"], st["matrix"], st["encoding"] = _host_pairs(made, False), _protein_matrix(), protein_encoding()
        else:
            # large batches sit in pinned memory, klign's strings and a short call's arrays do not
            p = st["pairs"] = _host_pairs(made, kind == "host" and case["n"] > 1000)
            if kind == "block":  # the C entry points take pointer arrays, as the C++ header hands them over
                st["reads"] = (p.a_seq.ctypes.data + p.a_off).astype(np.uint64)
                st["windows"] = (p.b_seq.ctypes.data + p.b_off).astype(np.uint64)
                st["longest"] = int(p.a_len.max()), int(p.b_len.max())
    torch.cuda.synchronize()
    return st


def _block(st):
    d, p = st["drv"], st["pairs"]
    args = (st["reads"].ctypes.data, p.a_len.ctypes.data, st["windows"].ctypes.data, p.b_len.ctypes.data, st["n"],
            *st["longest"])
    for call in (d._lib.mhsw_run_kernel_forwards, d._lib.mhsw_run_kernel_backwards):
        if call(d._h, *args) != 0:
            raise RuntimeError(d._lib.mhsw_driver_last_error(d._h).decode())
        d.kernel_block()
    r = d.get_aln_results()
    return [r.top_scores32, r.query_begin32, r.query_end32, r.ref_begin32, r.ref_end32, r.top_scores, r.query_begin,
            r.query_end, r.ref_begin, r.ref_end]


def _cigars(st):
    """The batch's CIGARs into the program's own arrays, by the C entry point."""
    d, total = st["drv"], C.c_int64(0)
    nops, mism, off, ops = st["cigars"]
    if d._lib.mhsw_last_cigar(d._h, nops.ctypes.data, mism.ctypes.data, off.ctypes.data, ops.ctypes.data,
                              ops.shape[0], C.byref(total), 1) != 0:
        raise RuntimeError(d._lib.mhsw_driver_last_error(d._h).decode())
    return st["cigars"]


def run(st):
    kind = st["kind"]
    if kind == "host":
        return st["drv"].align_pairs(st["pairs"], st["form"])
    if kind == "block":
        return _block(st)
    if kind == "device":
        st["drv"].align_pairs_device(st["dev"], st["out"].data_ptr(), st["form"])
        if st["mode"] == "score2":
            return [st["out"], st["drv"].last_score2(st["n"])]
        if st["mode"] == "cigar":
            return [st["out"], *_cigars(st)]
        return st["out"]
    if kind == "klign":
        return klign_align(st["drv"], st["contigs"], st["cand"])
    if kind == "serving":
        out5, win, _ = st["srv"].wait(st["srv"].submit(st["req"]))
        return [out5, win]
    if kind == "protein":
        return st["drv"].align_protein(st["pairs"], st["matrix"], st["encoding"])
    forward_noalloc(st["dev"], st["out"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    return st["out"]


# Mean extents of the mixes (A, B and A times B), for the work of a pass.
_MEAN = {"fixed": (150, 300, 45000), "mix": (175, 570, 102000), "uneven": (175, 475, 83000),
         "longref": (250, 5120, 1280000), "longpair": (4430, 4430, 2.9e7)}


def work(case):
    """Bytes: sequences, offsets, lengths and results once.  Operations: six integer ones a
    forward cell (two gap updates, the diagonal sum, the three-way and zero maxima)."""
    n, kind = case["n"], case["kind"]
    if kind == "klign":  # the 60% inexact reads against windows of about their own length
        return {"bytes": n * (2 * 175 + 8 + 17 + 34), "flops": 6.0 * 0.6 * n * 32400}
    if kind == "serving":
        return {"bytes": n * (175 + 560 + 24 + 28), "flops": 6.0 * n * 175 * 560}
    if kind == "protein":
        m = (case["lo"] + case["hi"]) / 2
        return {"bytes": n * (2 * m + 24 + 20), "flops": 6.0 * n * m * m}
    a, b, cells = _MEAN[case["mix"]]
    return {"bytes": n * (a + b + 24 + (12 if kind == "noalloc" else 20)), "flops": 6.0 * n * cells}


# ---- the same results by plain tensor code, in 64 bits ---------------------------------

def _padded(arena, off, lens, codes):
    width = max(1, int(lens.max()))
    t = torch.arange(width, device=DEV)
    ok = t[None, :] < lens[:, None]
    idx = torch.where(ok, off[:, None] + t[None, :], 0)
    return torch.where(ok, codes[arena[idx].long()], codes[256])


def _best_cell(a, b, table, go, ge):
    """(score, row, column) of the largest cell, smallest row and then column among equals;
    a and b are padded code matrices, table[a, b] the scores (padding scores far below 0)."""
    n, m = a.shape
    k = b.shape[1]
    low = -(1 << 40)
    pad = torch.full((n, m), table.shape[0] - 1, dtype=b.dtype, device=DEV)
    back = torch.cat([pad, b, pad], 1).flip(1)
    h1 = torch.zeros((n, m + 1), dtype=torch.int64, device=DEV)
    h2 = torch.zeros_like(h1)
    e = torch.full_like(h1, low)
    f = torch.full_like(h1, low)
    key = torch.zeros((n, m), dtype=torch.int64, device=DEV)
    row = torch.arange(m, device=DEV)
    arow = a * table.shape[0]
    flat = table.reshape(-1)
    for d in range(m + k - 1):
        s = m + k - 1 - d
        col = back[:, s:s + m]          # column d - i at row i
        ne = torch.maximum(e[:, :-1] - ge, h1[:, :-1] - go)
        nf = torch.maximum(f[:, 1:] - ge, h1[:, 1:] - go)
        h = torch.maximum(torch.maximum(h2[:, :-1] + flat[arow + col], torch.maximum(ne, nf)), torch.zeros_like(ne))
        inside = (d - row >= 0) & (d - row < k)
        h = torch.where(inside, h, 0)
        h2, h1 = h1, torch.nn.functional.pad(h, (1, 0))
        e, f = (torch.nn.functional.pad(torch.where(inside, x, low), (1, 0), value=low) for x in (ne, nf))
        key = torch.maximum(key, torch.where(h > 0, (h << 40) | ((0xFFFFF - row) << 20) | (0xFFFFF - (d - row)), 0))
    best = key.amax(1)
    return best >> 40, 0xFFFFF - ((best >> 20) & 0xFFFFF), 0xFFFFF - (best & 0xFFFFF)


def _exact_pairs(p, codes, table, go, ge, begins=True):
    a, ao, al, b, bo, bl = p
    n = al.shape[0]
    if float((al.double() * bl.double()).sum()) > 4e9 or int(al.max()) + int(bl.max()) > 6000:
        return None
    out = torch.zeros((n, 5), dtype=torch.int64, device=DEV)
    order = torch.argsort(al * 4096 + bl)
    for i in range(0, n, 8192):
        q = order[i:i + 8192]
        s, ie, je = _best_cell(_padded(a, ao[q], al[q], codes), _padded(b, bo[q], bl[q], codes), table, go, ge)
        hit = s > 0
        ie, je = torch.where(hit, ie, -1), torch.where(hit, je, 0)
        ib, jb = torch.full_like(ie, -1), torch.zeros_like(je)
        if begins and bool(hit.any()):
            qa, ra = _padded(a, ao[q], al[q], codes), (ie + 1).clamp(min=1)
            qb, rb = _padded(b, bo[q], bl[q], codes), (je + 1).clamp(min=1)

            def turned(x, k):
                t = torch.arange(int(k.max()), device=DEV)
                idx = (k[:, None] - 1 - t[None, :])
                return torch.where(idx >= 0, torch.gather(x, 1, idx.clamp(min=0)), table.shape[0] - 1)

            _, ri, rj = _best_cell(turned(qa, ra), turned(qb, rb), table, go, ge)
            ib, jb = torch.where(hit, ie - ri, ib), torch.where(hit, je - rj, jb)
        out[q] = torch.stack([s, ib, ie, jb, je], 1)
    return out


def _dna_tables(scores):
    m, x, _, _, amb = scores
    codes = torch.full((257,), 4, dtype=torch.int64, device=DEV)
    for k, pair in enumerate((b"Aa", b"Cc", b"Gg", b"Tt")):
        for c in pair:
            codes[c] = k
    codes[256] = 5
    table = torch.full((6, 6), -(1 << 30), dtype=torch.int64, device=DEV)
    table[:5, :5] = -x
    table[torch.arange(4), torch.arange(4)] = m
    table[4, :5] = table[:5, 4] = -amb
    return codes, table


def exact(case, seed):
    kind = case["kind"]
    if kind == "klign":
        return None
    made = _inputs(case, seed)
    scores = _scores(case)
    if kind == "protein":
        enc = protein_encoding()
        codes = torch.full((257,), 22, dtype=torch.int64, device=DEV)
        codes[:91] = torch.from_numpy(enc.astype(np.int64)).to(DEV)
        codes[256] = 24
        table = torch.full((25, 25), -(1 << 30), dtype=torch.int64, device=DEV)
        table[:24, :24] = torch.from_numpy(_protein_matrix().astype(np.int64)).to(DEV)
        return _exact_pairs(made, codes, table, 11, 1)
    codes, table = _dna_tables(scores)
    _, _, go, ge, _ = scores
    if kind == "serving":
        (arena, off, ln), req = made
        cid, pos, la = (torch.from_numpy(x.astype(np.int64)).to(DEV) for x in (req.cid, req.pos, req.len))
        ws = (pos - FLANK).clamp(min=0)
        we = torch.minimum(ln[cid], pos + la + FLANK)
        a = torch.from_numpy(req.seq).to(DEV)
        out5 = _exact_pairs((a, torch.from_numpy(req.off).to(DEV), la, arena, off[cid] + ws, we - ws), codes, table,
                            go, ge)
        return None if out5 is None else [out5, ws]
    out5 = _exact_pairs(made, codes, table, go, ge, kind != "noalloc")
    if out5 is None:
        return None
    if kind == "noalloc":
        return out5[:, [0, 2, 4]].contiguous()
    if kind == "block":
        cols = [out5[:, k].contiguous() for k in range(5)]
        return cols + cols
    mode = case.get("mode", "plain")
    return out5 if mode == "plain" else [out5, None] if mode == "score2" else [out5, None, None, None, None]
