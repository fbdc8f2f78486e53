"""What is measured: the alignment work a read mapper hands to this framework.

Each case is one pass of a public entry point over inputs of the kind that
entry point meets in a mapping run: reads cut from their windows with 1 %
substitutions, 0.1 % indels of 1-3 bases and A-to-G editing at 5 % of the
reference A's (T-to-C on reverse-strand reads), a few N runs where a case
says so.  Device batches keep their inputs and outputs on the GPU, as a
pipeline that streams batches through resident buffers does; one handle
serves every batch, as one worker keeps one handle.

Kinds (the "kind" of a case):
  call    one extend_hint call on ASCII bytes, as a per-read caller makes it
  band    esp_batch_extend_device, banded (half < 0: the whole matrix, which
          is what extend() runs)
  hint    esp_batch_extend_device, the two-attempt extend_hint policy
  myers   esp_batch_myers_device (mode 0 best end, 1 best start, 2 global)
  myers_host  batch.myers_batch_host: host arrays in, host array out
  splice  esp_batch_splice_device: channel A over split reads and their
          library candidates on a resident genome

All outputs are whole numbers.  A CIGAR row is defined up to its record's
n_ops (and only when the record's status is 0), so run() returns the rows
with the entries after that as zeros.
"""
import ctypes
import math

import numpy as np
import torch

from esperanto_gb300 import _native
from esperanto_gb300 import batch as B
from esperanto_gb300 import split as S
from esperanto_gb300.extend import (INITIAL_BAND, OP_CHARS, DiagHint, EditDir, ExtendBuffer, ExtendParams,
                                    extend_hint)

STRIDE = 32          # CIGAR slots a pair, as the benchmark's batches have
MIXED = ((16, .4), (32, .3), (64, .2), (128, .1))  # band halves of the mixed-length batch
DP_OPS = 18          # integer operations of one DP cell's recurrence
MYERS_OPS = 10 / 32  # of one bit-parallel cell
HINT_HALF = INITIAL_BAND
ESCALATES = 0.46     # share of reads whose band touch sends them to the full matrix


def listed():
    return [
        # one read from a per-read caller: the smallest call there is
        dict(name="call_hint_150", kind="call", lo=150, hi=150, half=32),
        # a worker's small chunk of reads (the warp-per-pair kernel's range)
        dict(name="band_1000_mixed", kind="band", n=1000, lo=50, hi=300, half=0, edit=0, ns=0),
        # fixed-length reads against read + 2 x 32 windows, one sequencer chunk
        dict(name="band_64k_150x214", kind="band", n=65536, lo=150, hi=150, half=32, edit=0, ns=0),
        # a ragged mid-size batch: trimmed reads, N runs, editing-aware scores
        dict(name="band_200k_mixed_n", kind="band", n=200003, lo=50, hi=300, half=0, edit=1, ns=1),
        # the large batch: trimmed reads of a whole lane slice
        dict(name="band_4m_mixed", kind="band", n=4194304, lo=50, hi=300, half=0, edit=0, ns=0),
        # extend(): whole windows, no band
        dict(name="full_16k", kind="band", n=16384, lo=50, hi=250, half=-1, edit=0, ns=0),
        # the policy a mapper calls, at the size one served request has
        dict(name="hint_64k_150x214", kind="hint", n=65536, lo=150, hi=150, half=32, edit=0, ns=0),
        # and over a large batch of trimmed reads
        dict(name="hint_1m_mixed", kind="hint", n=1048576, lo=50, hi=300, half=0, edit=0, ns=0),
        # the edit-distance filter ahead of the DP
        dict(name="myers_1m_150x200", kind="myers", n=1048576, mode=0, lo=150, hi=150, slack=50),
        # the same filter looking for starts, reads of every length it takes
        dict(name="myers_100k_start", kind="myers", n=100003, mode=1, lo=20, hi=256, slack=100),
        # the filter called on host arrays, copies included
        dict(name="myers_host_256k", kind="myers_host", n=262144, mode=0, lo=150, hi=150, slack=50),
        # rescue of reads split over a junction, all their candidates
        dict(name="splice_64k", kind="splice", n=65536, length=150),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "band", "band", "band", "hint", "hint", "myers", "myers", "myers_host",
                       "splice"])
    if kind == "call":
        n = rng.randint(50, 300)
        return dict(kind=kind, lo=n, hi=n, half=rng.choice([16, 32, 64]))
    if kind in ("band", "hint"):
        lo = rng.randint(50, 150)
        hi = rng.choice([lo, rng.randint(lo, 300)])
        half = rng.choice([0, 0, 16, 32, 64, 128] + ([-1] if kind == "band" else []))
        most = {"band": 2000000, "hint": 600000}[kind] // (4 if half in (-1, 128) else 1)
        return dict(kind=kind, n=_log_int(rng, 100, most), lo=lo, hi=hi, half=half,
                    edit=rng.choice([0, 1, 2]), ns=rng.choice([0, 1]))
    if kind in ("myers", "myers_host"):
        lo = rng.randint(20, 200)
        hi = rng.choice([lo, rng.randint(lo, 256)])
        return dict(kind=kind, n=_log_int(rng, 500, 2000000), mode=rng.choice([0, 1, 2]), lo=lo,
                    hi=hi, slack=rng.randint(10, 120))
    return dict(kind=kind, n=_log_int(rng, 100, 50000), length=rng.randint(80, 200))


# ---- inputs, made on the GPU from the seed ---------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _randint(g, lo, hi, shape, dtype=torch.int64):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _starts(lens):
    return torch.cumsum(lens, 0) - lens


def _derive(g, codes, read_pos, lens, src, limit, fwd):
    """Write reads into `codes` at read_pos: bases of codes[src ...] (never at
    or past `limit`) with the error model above."""
    for a in range(0, len(lens), 1 << 18):
        ln = lens[a:a + (1 << 18)]
        first = _starts(ln)
        total = int(ln.sum())
        pid = torch.repeat_interleave(torch.arange(len(ln), device="cuda"), ln)
        k = torch.arange(total, device="cuda") - first[pid]
        at = read_pos[a:a + (1 << 18)][pid] + k
        u = _rand(g, total)
        size = 1 + (_rand(g, total) < .5).long() + (_rand(g, total) < .25).long()
        ins, dele = u < .0005, (u >= .0005) & (u < .001)
        shift = torch.cumsum(torch.where(ins, -size, torch.where(dele, size, 0)), 0)
        shift = shift - shift[first[pid]]
        drawn = ins.clone()
        for d in (1, 2):
            drawn[d:] |= ins[:-d] & (size[:-d] > d)
        s = src[a:a + (1 << 18)][pid] + k + shift
        drawn |= (s < 0) | (s >= limit[a:a + (1 << 18)][pid])
        c = torch.where(drawn, codes[at], codes[torch.where(drawn, at, s)])
        v = _rand(g, total)
        c = torch.where(v < .01, (c + 1 + _randint(g, 0, 3, (total,), torch.uint8)) & 3, c)
        edit = (v >= .01) & (v < .06)
        f = fwd[a:a + (1 << 18)][pid]
        c = torch.where(edit & f & (c == 0), 2, torch.where(edit & ~f & (c == 3), 1, c))
        codes[at] = c.to(torch.uint8)


def _pack(codes):
    pad = torch.zeros((-len(codes)) % 4 + 64, dtype=torch.uint8, device="cuda")
    q = torch.cat([codes, pad]).view(-1, 4)
    return (q[:, 0] << 6) | (q[:, 1] << 4) | (q[:, 2] << 2) | q[:, 3]


def _u64(x):
    return [(x & 0xffffffff), x >> 32]


def _records(cols):
    """int64 columns -> int32 records (values taken as unsigned)."""
    t = torch.stack([c.expand(len(cols[0])) if c.dim() == 0 else c for c in cols], 1)
    return torch.where(t > 0x7fffffff, t - (1 << 32), t).to(torch.int32).contiguous()


def _n_runs(g, lens, share):
    """At most one N run of 1-4 bases a sequence, on `share` of them."""
    has = _rand(g, len(lens)) < share
    start = (_rand(g, len(lens)) * (lens - 4)).long().clamp(min=0)
    return has, start, start + 1 + _randint(g, 0, 4, (len(lens),))


def _lens(g, n, lo, hi):
    return _randint(g, lo, hi + 1, (n,))


def _halves(g, n, half):
    if half != 0:
        return torch.full((n,), half, dtype=torch.int64, device="cuda")
    u, out, acc = _rand(g, n), torch.zeros(n, dtype=torch.int64, device="cuda"), 0.
    for h, p in MIXED:
        out = torch.where((u >= acc) & (u < acc + p + 1e-6), h, out)
        acc += p
    return torch.where(out == 0, MIXED[-1][0], out)


def _pairs(seed, n, lo, hi, half, ns):
    """Reads against the windows they come from: arena, pair records, N runs."""
    g = _gen(seed)
    lens = _lens(g, n, lo, hi)
    half = _halves(g, n, half)
    flank = torch.where(half < 0, 50, half)  # no band: 50 bases on either side
    wins = lens + 2 * flank
    read_pos = _starts(lens + wins)
    win_pos = read_pos + lens
    codes = _randint(g, 0, 4, (int((lens + wins).sum()),), torch.uint8)
    _derive(g, codes, read_pos, lens, win_pos + flank, win_pos + wins, _rand(g, n) < .5)
    zero = torch.zeros(n, dtype=torch.int64, device="cuda")
    iv, n_first, counts = torch.zeros((0, 2), dtype=torch.int32, device="cuda"), zero, zero
    if ns:
        runs = [_n_runs(g, lens, .01), _n_runs(g, wins, .005)]
        counts = runs[0][0].long() | (runs[1][0].long() << 16)
        per = runs[0][0].long() + runs[1][0].long()
        n_first = _starts(per)
        iv = torch.zeros((int(per.sum()), 2), dtype=torch.int32, device="cuda")
        for q, (has, s, e) in enumerate(runs):
            at = (n_first + (runs[0][0].long() if q else 0))[has]
            iv[at, 0], iv[at, 1] = s[has].int(), e[has].int()
    pairs = _records(_u64(read_pos) + _u64(win_pos) +
                     [lens, wins, flank, half & 0xffffffff, n_first, counts])
    return _pack(codes), pairs, iv, int(lens.max()), int(wins.max()), int(half.max())


def _myers_pairs(seed, n, mode, lo, hi, slack):
    """Queries against texts that hold them (one in ten does not)."""
    g = _gen(seed)
    lens = _lens(g, n, lo, hi)
    room = torch.full_like(lens, slack)
    texts = lens + (room if mode != 2 else _randint(g, 0, 9, (n,)))
    read_pos = _starts(lens + texts)
    text_pos = read_pos + lens
    codes = _randint(g, 0, 4, (int((lens + texts).sum()),), torch.uint8)
    src = text_pos + (_rand(g, n) * (texts - lens + 1)).long()
    src = torch.where(_rand(g, n) < .1, 1 << 60, src)  # past the limit: unrelated
    _derive(g, codes, read_pos, lens, src, text_pos + texts, _rand(g, n) < .5)
    zero = torch.zeros(n, dtype=torch.int64, device="cuda")
    pairs = _records(_u64(read_pos) + _u64(text_pos) + [lens, texts, zero, zero])
    return _pack(codes), pairs, int(lens.max())


def _split_reads(seed, n, length):
    """Reads across planted GT..AG junctions, eight a locus, each with the
    locus's true junction and its decoys as candidates in library order."""
    g = _gen(seed)
    loci = (n + 7) // 8
    flank = 2 * length
    intron = torch.exp(math.log(60) + _rand(g, loci) * math.log(50000 / 60)).long()
    clen = 2 * flank + intron
    stride = (clen + 3) // 4 * 4
    base = _starts(stride)
    codes = _randint(g, 0, 4, (int(stride.sum()),), torch.uint8)
    off = torch.tensor([k for k in range(-20, 21) if k], device="cuda")
    donor, acceptor = _rand(g, loci, 40) < 1 / 16, _rand(g, loci, 40) < 1 / 16
    for mask, at, two in ((donor, base + flank, (0, 2, 3)), (acceptor, base + flank + intron, (-2, 0, 2))):
        rows, cols = torch.nonzero(mask, as_tuple=True)
        for p in (at[rows] + off[cols], at):  # decoys, then the true site over them
            codes[p + two[0]], codes[p + two[0] + 1] = two[1], two[2]
    read_locus = torch.arange(n, device="cuda") // 8
    # spliced source of each locus: the exon ends, joined, in a scratch arena
    k = torch.arange(flank, device="cuda")
    joined = torch.cat([codes[(base + flank - flank // 2)[:, None] + k[:flank // 2]],
                        codes[(base + flank + intron)[:, None] + k[:flank // 2]]], 1).reshape(-1)
    cut = _randint(g, 20, length - 19, (n,))
    lens = torch.full((n,), length, dtype=torch.int64, device="cuda")
    work = torch.cat([joined, _randint(g, 0, 4, (n * length,), torch.uint8)])
    src = read_locus * (flank // 2 * 2) + flank // 2 - cut
    rpos = len(joined) + torch.arange(n, device="cuda") * length
    _derive(g, work, rpos, lens, src, (read_locus + 1) * (flank // 2 * 2),
            torch.ones(n, dtype=torch.bool, device="cuda"))
    reads_arena = _pack(work[len(joined):])
    tail = (cut + _randint(g, -3, 4, (n,))).clamp(1, length - 1)
    # candidates sorted by (start, end): donors before, the true start, donors after
    mask = torch.cat([donor[:, :20], acceptor[:, :20], torch.ones(loci, 1, dtype=torch.bool, device="cuda"),
                      acceptor[:, 20:], donor[:, 20:]], 1)
    z = torch.zeros(20, dtype=torch.int64, device="cuda")
    d_off = torch.cat([off[:20], z, z[:1], z, off[20:]])
    a_off = torch.cat([z, off[:20], z[:1], off[20:], z])
    rows, cols = torch.nonzero(mask[read_locus], as_tuple=True)
    locus = read_locus[rows]
    start, end = flank + d_off[cols], (flank + intron)[locus] + a_off[cols]
    support = torch.where(cols == 40, 5, 1 + _randint(g, 0, 3, (len(cols),)))
    cands = _records([locus, start, end, torch.zeros_like(locus), support])
    count = torch.bincount(rows, minlength=n)
    zero = torch.zeros(n, dtype=torch.int64, device="cuda")
    reads = _records(_u64(torch.arange(n, device="cuda") * length) +
                     [lens, tail, read_locus, zero, _starts(count), count, zero, zero])
    contigs = np.zeros(loci, S.CONTIG_DTYPE)
    contigs["base"], contigs["len"] = base.cpu().numpy(), clen.cpu().numpy()
    return _pack(codes).cpu().numpy(), contigs, reads_arena, reads, cands


_worker = {}


def _handle():
    """The worker's handle and its stream."""
    if not _worker:
        buf = ExtendBuffer()
        _worker["buf"] = buf
        _worker["stream"] = torch.cuda.ExternalStream(buf.stream_ptr())
    return _worker["buf"], _worker["stream"]


def _ascii(arena, pos, n):
    return B._ASCII[B.unpack_codes(arena, pos, n)].tobytes()


def prepare(case, seed):
    kind = case["kind"]
    buf, stream = _handle()
    st = dict(kind=kind, buf=buf, stream=stream)
    if kind == "call":
        arena, pairs, _, _, _, _ = _pairs(seed, 1, case["lo"], case["hi"], case["half"], 0)
        arena, p = arena.cpu().numpy(), pairs.cpu().numpy().view(B.PAIR_DTYPE).reshape(-1)[0]
        st.update(read=_ascii(arena, int(p["read_pos"]), int(p["read_len"])),
                  window=_ascii(arena, int(p["win_pos"]), int(p["win_len"])),
                  params=ExtendParams(), hint=DiagHint(case["half"]))
        return st
    n = case["n"]
    if kind in ("band", "hint"):
        arena, pairs, iv, m, w, half = _pairs(seed, n, case["lo"], case["hi"], case["half"], case["ns"])
        half = HINT_HALF if kind == "hint" else half
        st.update(n=n, arena=arena, pairs=pairs, iv=iv, mode=B.MODE_HINT if kind == "hint" else B.MODE_BAND,
                  limits=_native.BatchLimitsC(m, w, half),
                  params=ExtendParams(edit_dir=EditDir(case["edit"]))._c(),
                  out=torch.zeros((n, B.EXT_DTYPE.itemsize // 4), dtype=torch.int32, device="cuda"),
                  cigar=torch.zeros((n, STRIDE), dtype=torch.int32, device="cuda"))
    elif kind in ("myers", "myers_host"):
        arena, pairs, m = _myers_pairs(seed, n, case["mode"], case["lo"], case["hi"], case["slack"])
        st.update(n=n, mode=case["mode"], max_len=m)
        if kind == "myers":
            st.update(arena=arena, pairs=pairs,
                      out=torch.zeros((n, B.MYERS_RES_DTYPE.itemsize // 4), dtype=torch.int32, device="cuda"))
        else:
            st.update(arena=arena.cpu().numpy(),
                      pairs=pairs.cpu().numpy().view(B.MYERS_PAIR_DTYPE).reshape(-1))
    else:
        garena, contigs, arena, reads, cands = _split_reads(seed, n, case["length"])
        st.update(n=n, genome=S.Genome(garena, contigs, buf=buf), arena=arena, reads=reads, cands=cands,
                  length=case["length"], splice=S.SpliceParams()._c(), params=ExtendParams()._c(),
                  out=torch.zeros((n, S.SPLICE_RES_DTYPE.itemsize // 4), dtype=torch.int32, device="cuda"),
                  cigar=torch.zeros((n, STRIDE), dtype=torch.int32, device="cuda"))
    if kind != "myers_host":
        st["slots"] = torch.arange(STRIDE, dtype=torch.int32, device="cuda")
    return st


def _rows(st, n_ops, status):
    """The CIGAR rows up to their n_ops (0 after that and where refused)."""
    used = torch.where(st["out"][:, status] == 0, st["out"][:, n_ops], 0)
    return torch.where(st["slots"] < used[:, None], st["cigar"], 0)


def run(st):
    kind, buf = st["kind"], st["buf"]
    if kind == "call":
        x, escalated = extend_hint(st["read"], st["window"], st["params"], buf, st["hint"],
                                     with_escalation=True)
        ops = [OP_CHARS.index(o) | (k << 4) for o, k in x.cigar]
        return np.array([x.score, x.read_start, x.read_end, x.ref_start, int(escalated)] + ops, np.int64)
    if kind == "myers_host":
        r = B.myers_batch_host(st["pairs"], st["arena"], None, st["mode"], buf)
        return [r["dist"], r["pos"].astype(np.int64), r["status"]]
    L = _native.lib()
    if kind == "myers":
        buf.check(L.esp_batch_myers_device(
            buf.handle, st["mode"], st["pairs"].data_ptr(), st["n"], st["max_len"], st["arena"].data_ptr(),
            st["arena"].numel(), None, 0, st["out"].data_ptr(), st["stream"].cuda_stream))
        return st["out"]
    with torch.cuda.stream(st["stream"]):
        if kind == "splice":
            buf.check(L.esp_batch_splice_device(
                buf.handle, st["genome"].handle, st["reads"].data_ptr(), st["n"], st["length"],
                st["arena"].data_ptr(), st["arena"].numel(), None, 0, st["cands"].data_ptr(),
                len(st["cands"]), ctypes.byref(st["splice"]), ctypes.byref(st["params"]),
                st["out"].data_ptr(), st["cigar"].data_ptr(), STRIDE, st["stream"].cuda_stream))
            return [st["out"], _rows(st, 6, 7)]
        iv = st["iv"]
        buf.check(L.esp_batch_extend_device(
            buf.handle, st["mode"], st["pairs"].data_ptr(), st["n"], st["arena"].data_ptr(),
            st["arena"].numel(), iv.data_ptr() if len(iv) else None, len(iv), ctypes.byref(st["limits"]),
            ctypes.byref(st["params"]), st["out"].data_ptr(), st["cigar"].data_ptr(), STRIDE,
            st["stream"].cuda_stream))
        return [st["out"], _rows(st, 4, 7)]


def work(case):
    """Expected cells of the case's distribution; every input read once,
    every result record and a short CIGAR written once."""
    kind = case["kind"]
    if kind == "splice":
        L, n = case["length"], case["n"]
        items = 6. * n                     # the true junction and about five decoys
        flanks = items * 11 * 2            # breakpoints x sides
        cells = flanks * L / 2 * (61 + ESCALATES * (L / 2 + 30))
        return dict(bytes=n * (L / 4 + 40 + 32 + 16) + items * 20, flops=cells * DP_OPS)
    m = (case["lo"] + case["hi"]) / 2
    m2 = m * m + ((case["hi"] - case["lo"] + 1) ** 2 - 1) / 12
    if kind in ("myers", "myers_host"):
        text = case["slack"] if case["mode"] != 2 else 4
        return dict(bytes=case["n"] * ((2 * m + text) / 4 + 32 + 16),
                    flops=case["n"] * (m2 + m * text) * MYERS_OPS)
    halves = MIXED if case["half"] == 0 else ((case["half"] if case["half"] > 0 else 50, 1.),)
    flank = sum(h * p for h, p in halves)
    if kind == "band" and case["half"] > -1:
        cells = m * (2 * flank + 1)
    elif kind == "band":
        cells = m2 + 2 * m * flank
    else:
        cells = m * (2 * HINT_HALF + 1) + ESCALATES * (m2 + 2 * m * flank)
    n = case.get("n", 1)
    return dict(bytes=n * ((2 * m + 2 * flank) / 4 + 40 + 32 + 16), flops=n * cells * DP_OPS)


def exact(case, seed):
    """Every output is a whole number and has to be equal: nothing to round."""
    return None
