"""Performance cases of the aligner: the calls its users make, through the public entry points.

A case is a dict of plain values; prepare() makes its inputs on the GPU machine from a seed, run()
makes one pass.  All data are synthetic, with the shapes and error rates of this repository's
configurations: references of uniform ACGT (the larger ones in 24 sequences of log-normal
length, 10 % of them copies of 300-base repeat units at 3 % divergence), reads with 1 %
substitutions and 0.1 % indels of 1-3 bases, 5 % of them random.

Kinds:
  align    Context.align_into: reads FASTA in pinned host memory to text records in pinned host
           memory on a resident index; with "format" 1 SAM records, with "seeder" 1 the
           command line's default seed-and-extend seeder
  cold     a whole command-line run in memory: index built from the reference FASTA, reads aligned
  paired   Context.align_paired_into: mate pairs
  pairs    swift_sw_pairs on device buffers: reads of 36-250 bases, each against 1-64 regions
  long     swift_sw_pairs on device buffers: queries of 1-4 kb against regions of 2-8 kb
  batch    swift_sw_batch on device buffers: n pairs of one query and window length
  serving  Server: a burst of requests of 1-10,000 reads of 50-300 bases
"""
import ctypes as C
import math

import numpy as np
import torch

import swift_gb300 as sg

DEV = "cuda"
ACGT = (65, 67, 71, 84)


def listed():
    return [
        # the smallest call: one read on a small genome, all latency and launches
        dict(name="one_read", kind="align", ref_bp=1_000_000, seqs=1, reads=1, len=100),
        # the repository's small configuration: a bacterial-size reference, 10,000 reads
        dict(name="small_10k", kind="align", ref_bp=1_000_000, seqs=1, reads=10_000, len=100),
        # its scale configuration, the headline benchmark: a sequencing run's chunk
        dict(name="scale_1m", kind="align", ref_bp=50_000_000, seqs=24, reads=1_000_000, len=100),
        # longer reads of odd length, beyond the reference program's 199 bases
        dict(name="reads_251", kind="align", ref_bp=50_000_000, seqs=24, reads=100_000, len=251),
        # a whole run of the command line: index built, then short odd reads aligned
        dict(name="cold_75", kind="cold", ref_bp=4_000_000, seqs=3, reads=20_000, len=75),
        # SAM output: every candidate alignment is traced and printed
        dict(name="sam_200k", kind="align", ref_bp=50_000_000, seqs=24, reads=200_000, len=100,
             format=1),
        # the command line's default seeder
        dict(name="lt13_200k", kind="align", ref_bp=20_000_000, seqs=24, reads=200_000, len=100,
             seeder=1),
        # paired-end reads
        dict(name="paired_100k", kind="paired", ref_bp=20_000_000, seqs=24, reads=100_000,
             len=100),
        # batched pairs of uneven lengths (the batched configuration)
        dict(name="pairs_uneven", kind="pairs", ref_bp=50_000_000, reads=20_000, regions=64),
        # long queries against long regions (the long-region configuration)
        dict(name="pairs_long", kind="long", ref_bp=50_000_000, reads=500),
        # the reference library's batch call on device buffers, as its pipeline makes it
        dict(name="batch_100x300", kind="batch", pairs=20_000, q=100, r=300),
        # serving: requests that arrive at once on a resident 200 Mbp reference
        dict(name="serving_48", kind="serving", ref_bp=200_000_000, seqs=24, requests=48,
             workers=4),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["align", "align", "align", "sam", "lt13", "cold", "paired", "pairs", "long",
                       "batch", "serving"])
    ref = log(1_000_000, 50_000_000)
    seqs = 1 if ref < 3_000_000 else rng.randint(2, 24)
    if kind == "align":
        return dict(kind="align", ref_bp=ref, seqs=seqs, reads=log(1, 400_000),
                    len=rng.randint(36, 250))
    if kind == "sam":
        return dict(kind="align", ref_bp=ref, seqs=seqs, reads=log(1, 100_000),
                    len=rng.randint(36, 199), format=1)
    if kind == "lt13":
        return dict(kind="align", ref_bp=min(ref, 20_000_000), seqs=seqs, reads=log(1, 100_000),
                    len=rng.randint(50, 199), seeder=1)
    if kind == "cold":
        return dict(kind="cold", ref_bp=log(1_000_000, 8_000_000), seqs=rng.randint(1, 8),
                    reads=log(100, 50_000), len=rng.randint(36, 199))
    if kind == "paired":
        return dict(kind="paired", ref_bp=min(ref, 20_000_000), seqs=seqs, reads=log(1, 80_000),
                    len=rng.randint(50, 150))
    if kind == "pairs":
        return dict(kind="pairs", ref_bp=ref, reads=log(50, 20_000), regions=rng.randint(4, 64))
    if kind == "long":
        return dict(kind="long", ref_bp=ref, reads=log(8, 500))
    if kind == "batch":
        q = rng.randint(20, 250)
        return dict(kind="batch", pairs=log(10, 20_000), q=q, r=rng.randint(q, 500))
    return dict(kind="serving", ref_bp=ref, seqs=seqs, requests=rng.randint(2, 48),
                workers=rng.choice([1, 2, 4]))


# ---------------------------------------------------------------------------
# inputs


class Rand:
    """Seeded draws on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def ints(self, lo, hi, n, dtype=torch.int64):
        return torch.randint(lo, hi, n if isinstance(n, tuple) else (n,), generator=self.g,
                             device=DEV, dtype=dtype)

    def unit(self, n):
        return torch.rand(n if isinstance(n, tuple) else (n,), generator=self.g, device=DEV)


def lut(values):
    return torch.tensor(values, dtype=torch.uint8, device=DEV)


def reference(r, total, n_seqs, repeats):
    """(base codes, sequence starts on the host with the end appended)."""
    codes = r.ints(0, 4, total, torch.uint8)
    if repeats:
        units = r.ints(0, 4, (500, 300), torch.uint8)
        slots = total // 300
        at = torch.randperm(slots, generator=r.g, device=DEV)[: int(round(0.1 * slots))]
        copies = units[r.ints(0, 500, len(at))]
        mutate = (r.unit(tuple(copies.shape)) < 0.03).to(torch.uint8)
        copies = (copies + mutate * r.ints(1, 4, tuple(copies.shape), torch.uint8)) % 4
        codes[: slots * 300].view(slots, 300)[at] = copies
    w = np.exp(0.8 * torch.randn(n_seqs, generator=r.g, device=DEV).cpu().numpy().astype(float))
    lens = np.maximum((w / w.sum() * total).astype(np.int64), 2000)
    lens[lens.argmax()] += total - lens.sum()
    return codes, np.concatenate([[0], np.cumsum(lens)])


def reference_fasta(codes, starts):
    letters = lut(ACGT)[codes.long()] if codes.numel() < (1 << 26) else torch.cat(
        [lut(ACGT)[c.long()] for c in codes.split(1 << 26)])
    out = []
    for i in range(len(starts) - 1):
        s = letters[starts[i]:starts[i + 1]]
        full = len(s) // 60
        lines = torch.full((full, 61), 10, dtype=torch.uint8, device=DEV)
        lines[:, :60] = s[: full * 60].view(full, 60)
        out.append(b">chr%d\n" % (i + 1))
        out.append(lines.cpu().numpy().tobytes())
        if len(s) % 60:
            out.append(s[full * 60:].cpu().numpy().tobytes() + b"\n")
    return b"".join(out)


def read_codes(r, codes, starts, n, length, random_share=0.05):
    """n x length base codes: reads from uniform positions, the error model applied."""
    st = torch.as_tensor(starts, device=DEV)
    pos = r.ints(0, int(starts[-1]), n)
    sid = torch.searchsorted(st, pos, right=True) - 1
    pos = torch.minimum(pos, st[sid + 1] - length - 4).clamp_(min=0)
    at = r.ints(0, length, n)
    size = r.ints(1, 4, n)
    what = r.unit(n)
    p = min(0.5, 0.001 * length)
    dele, ins = what < p / 2, (what >= p / 2) & (what < p)
    is_random = r.unit(n) < random_share
    out = torch.empty((n, length), dtype=torch.uint8, device=DEV)
    k = torch.arange(length, device=DEV)
    for lo in range(0, n, 250_000):
        hi = min(n, lo + 250_000)
        c = slice(lo, hi)
        a, z = at[c, None], size[c, None]
        src = k + torch.where(dele[c, None] & (k >= a), z, 0)
        src = src - torch.where(ins[c, None] & (k >= a + z), z, 0)
        b = codes[(pos[c, None] + src).clamp_(max=int(starts[-1]) - 1)]
        b = (b + (r.unit((hi - lo, length)) < 0.01) * r.ints(1, 4, (hi - lo, length), torch.uint8)) % 4
        fresh = (ins[c, None] & (k >= a) & (k < a + z)) | is_random[c, None]
        out[c] = torch.where(fresh, r.ints(0, 4, (hi - lo, length), torch.uint8), b)
    return out


def reads_fasta(rows, suffix=b""):
    """FASTA bytes (device) of rows of letters, the reads named r0, r1, ..."""
    n, length = rows.shape
    parts, lo = [], 0
    for d in range(1, 9):
        hi = min(n, 10 ** d)
        if hi <= lo:
            break
        w = 2 + d + len(suffix) + 1
        m = torch.full((hi - lo, w + length + 1), 10, dtype=torch.uint8, device=DEV)
        m[:, 0], m[:, 1] = ord(">"), ord("r")
        num = torch.arange(lo, hi, device=DEV)
        for t in range(d):
            m[:, 1 + d - t] = (48 + num // 10 ** t % 10).to(torch.uint8)
        for t, c in enumerate(suffix):
            m[:, 2 + d + t] = c
        m[:, w:w + length] = rows[lo:hi]
        parts.append(m.reshape(-1))
        lo = hi
    return torch.cat(parts)


def pinned(t):
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(t)
    return h


def ragged(lens):
    """(offsets, row of every element, place in its row) of rows of the given lengths."""
    off = torch.cumsum(lens, 0) - lens
    row = torch.repeat_interleave(torch.arange(len(lens), device=DEV), lens)
    return off, row, torch.arange(len(row), device=DEV) - off[row]


def edited(r, codes, pos, lens, sub, indel):
    """Concatenated letters of len(lens) queries from pos on, with substitutions and indels of
    1-3 bases, and their offsets."""
    off, row, k = ragged(lens)
    u = r.unit(len(row))
    skip = torch.where(u < indel / 2, r.ints(1, 4, len(row)), 0)
    ins = (u >= indel / 2) & (u < indel)
    grown = torch.cumsum(skip - ins.long(), 0)
    first = grown[off] - (skip - ins.long())[off]
    src = pos[row] + k + grown - first[row]
    b = codes[src.clamp_(0, len(codes) - 1)]
    b = (b + (r.unit(len(row)) < sub) * r.ints(1, 4, len(row), torch.uint8)) % 4
    b = torch.where(ins, r.ints(0, 4, len(row), torch.uint8), b)
    return lut(ACGT)[b.long()], off


# ---------------------------------------------------------------------------
# prepare / run


def params_of(case, index):
    kw = dict(seed_len=index.seed_len, ignore_thres=index.ignore_thres)
    if case.get("format"):
        kw["out_format"] = case["format"]
    if case.get("seeder"):
        kw["seeder"] = case["seeder"]
    if case.get("len", 0) > 199:
        kw["max_read_len"] = 300
    return sg.default_params(**kw)


def one_read(codes):
    return lut(ACGT)[codes[1000:1060].long()].cpu().numpy().tobytes()


def out_buffer(case, reads):
    """Pinned room for the text; all of it is returned, zero past the text's end."""
    per = 6 * (110 + 2 * case["len"]) if case.get("format") else 210 + 4 * case["len"]
    return torch.zeros(reads * per + 65536, dtype=torch.uint8, pin_memory=True)


def prepare(case, seed):
    r = Rand(seed * 7919 + 17)
    kind = case["kind"]
    ctx = sg.Context()
    if kind in ("align", "cold", "paired", "serving"):
        codes, starts = reference(r, case["ref_bp"], case["seqs"], case["ref_bp"] >= 10_000_000)
        fasta = reference_fasta(codes, starts)
    else:
        codes = r.ints(0, 4, case.get("ref_bp", 1_000_000), torch.uint8)
    s = dict(kind=kind, ctx=ctx)
    if kind in ("align", "cold"):
        n = case["reads"]
        share = 0.05 if n >= 1000 else 0.0
        rows = lut(ACGT)[read_codes(r, codes, starts, n, case["len"], share).long()]
        s["reads"] = pinned(reads_fasta(rows))
        s["out"] = out_buffer(case, n)
        if kind == "align":
            s["index"] = ctx.index(fasta)
            s["params"] = params_of(case, s["index"])
            if case.get("seeder"):
                # the index's tables for this seeder are made by the first call that wants them
                ctx.align(s["index"], b">r0\n" + one_read(codes) + b"\n", s["params"])
        else:
            s["fasta"] = fasta
    elif kind == "paired":
        n, length = case["reads"], case["len"]
        frag = r.ints(max(200, length), 501, n)
        st = torch.as_tensor(starts, device=DEV)
        pos = r.ints(0, int(starts[-1]), n)
        sid = torch.searchsorted(st, pos, right=True) - 1
        pos = torch.minimum(pos, st[sid + 1] - frag)
        k = torch.arange(length, device=DEV)
        mates = [codes[pos[:, None] + k], 3 - codes[(pos + frag - 1)[:, None] - k]]
        for t, m in enumerate(mates):
            m = (m + (r.unit((n, length)) < 0.01) * r.ints(1, 4, (n, length), torch.uint8)) % 4
            s["reads%d" % (t + 1)] = pinned(reads_fasta(lut(ACGT)[m.long()], b"/%d" % (t + 1)))
        s["out"] = out_buffer(case, 2 * n)
        s["index"] = ctx.index(fasta)
        one = one_read(codes) + b"\n"
        # as above: paired-end positions are made by the first paired call
        ctx.align_paired(s["index"], b">r0/1\n" + one, b">r0/2\n" + one)
    elif kind == "serving":
        # the requests' sizes are the case's, their reads the seed's
        g = np.random.default_rng(case["requests"])
        sizes = np.exp(g.uniform(0.0, math.log(10_000), case["requests"])).astype(int)
        lens = g.integers(50, 301, case["requests"])
        s["requests"] = []
        s["replies"] = [torch.zeros((int(n) + 32) * (230 + 4 * int(m)), dtype=torch.uint8)
                        for n, m in zip(sizes, lens)]
        for n, length in zip(sizes, lens):
            rows = lut(ACGT)[read_codes(r, codes, starts, int(n), int(length), 0.0).long()]
            s["requests"].append(reads_fasta(rows).cpu().numpy().tobytes())
        s["index"] = ctx.index(fasta)
        s["server"] = sg.Server(s["index"], workers=case["workers"],
                                params=sg.default_params(max_read_len=300))
    elif kind in ("pairs", "long"):
        n = case["reads"]
        if kind == "pairs":
            lens = r.ints(36, 251, n)
            pos = r.ints(0, len(codes) - 1000, n)
            letters, off = edited(r, codes, pos, lens, 0.01, 0.001)
            # 1 .. regions of them, as many of each
            regions = torch.arange(n, device=DEV) % case["regions"] + 1
            regions = regions[torch.randperm(n, generator=r.g, device=DEV)]
            _, read, k = ragged(regions)
            p = torch.where(k == 0, pos[read],
                            r.ints(0, len(codes) - 1000, len(read)))
            lo = (p - 64).clamp_(min=0)
            hi = torch.minimum(p + lens[read] + 64, torch.tensor(len(codes), device=DEV))
            ql, qo, ro, rl = lens[read], off[read], lo, hi - lo
        else:
            lens = r.ints(1000, 4001, n)
            least = torch.maximum(lens + 200, torch.tensor(2000, device=DEV))
            rl = least + (r.unit(n).double() * (8001 - least)).long()
            pos = r.ints(8000, len(codes) - 12_000, n)
            letters, qo = edited(r, codes, pos, lens, 0.03, 0.005)
            ro = pos - (r.unit(n).double() * (rl - lens)).long()
            ql = lens
        s["q"], s["r"] = letters, lut(ACGT)[codes.long()]
        s["qo"], s["ro"] = qo.contiguous(), ro.contiguous()
        s["ql"], s["rl"] = ql.to(torch.int32), rl.to(torch.int32)
        cs = 4000 + 8000 + 4 if kind == "long" else 0
        s["cs"] = cs
        m = len(ql)
        s["out"] = [torch.zeros(m, dtype=torch.int32, device=DEV) for _ in range(4)]
        # long alignments with their strings, the many short ones coordinates only
        s["cons"] = [torch.zeros((m, cs), dtype=torch.uint8, device=DEV) for _ in range(2 if cs else 0)]
    else:
        n, q, w = case["pairs"], case["q"], case["r"]
        pos = r.ints(w, len(codes) - w - 8, n)
        k = torch.arange(w + 1, device=DEV)
        windows = lut(ACGT)[codes[pos[:, None] + k].long()]
        # a few windows run into N, as at the edges of assembled sequence
        cut = torch.where(r.unit(n) < 0.005, r.ints(1, w + 1, n), w + 1)
        windows = torch.where(k >= cut[:, None], torch.tensor(78, dtype=torch.uint8, device=DEV), windows)
        # a quarter of the pairs are a read at its origin, the others chance hits
        true = r.unit(n) < 0.25
        frm = torch.where(true, pos + (r.unit(n).double() * max(w - q, 1)).long(),
                          r.ints(0, len(codes) - q - 8, n))
        letters, off = edited(r, codes, frm, torch.full((n,), q, device=DEV), 0.01, 0.001)
        queries = torch.zeros((n, q + 1), dtype=torch.uint8, device=DEV)
        queries[:, :q] = letters.view(n, q)
        windows[:, w] = 0
        s["q"], s["w"], s["Q"], s["R"] = queries, windows.contiguous(), q, w
        s["score"] = torch.zeros(n, dtype=torch.float32, device=DEV)
        s["out"] = [torch.zeros(n, dtype=torch.int32, device=DEV) for _ in range(3)]
        s["cons"] = [torch.zeros((n, q + w + 2), dtype=torch.uint8, device=DEV) for _ in range(2)]
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "align":
        n, _ = ctx.align_into(s["index"], s["reads"].data_ptr(), s["reads"].numel(),
                              s["out"].data_ptr(), s["out"].numel(), s["params"])
        return {"text": s["out"], "bytes": n}
    if kind == "cold":
        index = ctx.index(s["fasta"])
        n, _ = ctx.align_into(index, s["reads"].data_ptr(), s["reads"].numel(),
                              s["out"].data_ptr(), s["out"].numel())
        index.close()
        return {"text": s["out"], "bytes": n}
    if kind == "paired":
        n, _ = ctx.align_paired_into(s["index"], s["reads1"].data_ptr(), s["reads1"].numel(),
                                     s["reads2"].data_ptr(), s["reads2"].numel(),
                                     s["out"].data_ptr(), s["out"].numel())
        return {"text": s["out"], "bytes": n}
    if kind == "serving":
        tickets = [s["server"].submit(q) for q in s["requests"]]
        for t, reply in zip(tickets, s["replies"]):
            text = s["server"].wait(t)[0]
            reply.numpy()[:len(text)] = np.frombuffer(text, dtype=np.uint8)
        return s["replies"]
    if kind in ("pairs", "long"):
        c = [t.data_ptr() for t in s["cons"]] or [None, None]
        ctx._check(sg.lib().swift_sw_pairs(
            ctx._h, s["q"].data_ptr(), s["qo"].data_ptr(), s["ql"].data_ptr(), s["r"].data_ptr(),
            s["ro"].data_ptr(), s["rl"].data_ptr(), len(s["ql"]), 2, -1, -10, -1,
            *[t.data_ptr() for t in s["out"]], c[0], c[1], s["cs"], 0, None))
        return dict(zip(("score", "start", "end", "len"), s["out"])) | (
            dict(zip(("qcons", "rcons"), s["cons"])))
    ctx._check(sg.lib().swift_sw_batch(
        ctx._h, s["q"].data_ptr(), s["w"].data_ptr(), s["Q"], s["R"], len(s["q"]),
        C.c_float(2), C.c_float(-1), C.c_float(-10), C.c_float(-1), s["score"].data_ptr(),
        *[t.data_ptr() for t in s["out"]], *[t.data_ptr() for t in s["cons"]]))
    return dict(zip(("start", "end", "len", "qcons", "rcons"), s["out"] + s["cons"]),
                score=s["score"])


# ---------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Bytes: inputs read once (the reference as 2-bit codes and 4-byte positions, one per 12
    bases; the FASTA bytes themselves where the index is built), outputs written once.  Operations:
    for explicit pairs the recurrence, 6 integer operations a cell; else one table lookup's hash,
    2 operations for every base of both strands."""
    kind = case["kind"]
    if kind in ("align", "cold", "paired"):
        n = case["reads"] * (2 if kind == "paired" else 1)
        length = case["len"]
        records = n * (4 if case.get("format") else 1)
        line = 45 + length // 2 if case.get("format") else 150 + 3 * (length + 4)
        ref = case["ref_bp"] * (1 if kind == "cold" else 1 / 4 + 4 / 12)
        # a pass looks at no more of a large reference than its reads can touch
        ref = min(ref, n * 2.0 * (length * 32 + 12 * 75) + (case["ref_bp"] if kind == "cold" else 0))
        return {"bytes": n * (length + 8) + records * line + ref, "flops": n * length * 4}
    if kind == "serving":
        n = case["requests"] * (10_000 - 1) / math.log(10_000)
        ref = min(case["ref_bp"] * (1 / 4 + 4 / 12), n * 2.0 * (175 * 32 + 12 * 75))
        return {"bytes": n * (183 + 150 + 3 * 179) + ref, "flops": n * 175 * 4}
    if kind == "pairs":
        m = case["reads"] * (case["regions"] + 1) / 2
        cells = m * (143 * 143 + 214 ** 2 / 12 + 143 * 128)
        return {"bytes": case["reads"] * 143 + m * (271 + 24 + 16), "flops": 6 * cells}
    if kind == "long":
        m = case["reads"]
        return {"bytes": m * (2500 + 5350 + 2 * 2600 + 40), "flops": 6 * m * 2500 * 5560}
    m, q, r = case["pairs"], case["q"], case["r"]
    return {"bytes": m * (3 * q + r + 16), "flops": 6 * m * q * r}


def exact(case, seed):
    """The scores of a batch in 64-bit arithmetic: the recurrence over anti-diagonals, a gap's
    penalty gap_ext where the neighbour itself was reached the same way, else gap_open."""
    if case["kind"] != "batch":
        return None
    s = prepare(case, seed)
    n, Q, R = len(s["q"]), s["Q"], s["R"]
    q, w = s["q"][:, :Q].long(), s["w"][:, :R].long()
    zero = torch.zeros((n, Q + 1), dtype=torch.int64, device=DEV)
    h1, h2, d1 = zero, zero, zero  # by row; directions 1 diagonal, 2 up, 3 left
    best = torch.zeros(n, dtype=torch.int64, device=DEV)
    rows = torch.arange(1, Q + 1, device=DEV)
    for d in range(2, Q + R + 1):
        col = d - rows
        ok = (col >= 1) & (col <= R)
        b = w[:, (col - 1).clamp(0, R - 1)]
        same = (q == b) | (q == 78) | (b == 78)
        diag = h2[:, :-1] + torch.where(same, 2, -1)
        up = h1[:, :-1] + torch.where(d1[:, :-1] == 2, -1, -10)
        left = h1[:, 1:] + torch.where(d1[:, 1:] == 3, -1, -10)
        h = diag.clamp(min=0)
        code = (diag > 0).long()
        code = torch.where(up > h, 2, code)
        h = torch.maximum(h, up)
        code = torch.where(left > h, 3, code)
        h = torch.maximum(h, left)
        new, cd = zero.clone(), zero.clone()
        new[:, 1:] = torch.where(ok, h, 0)
        cd[:, 1:] = torch.where(ok, code, 0)
        best = torch.maximum(best, new.max(1).values)
        h1, h2, d1 = new, h1, cd
    return {"start": None, "end": None, "len": None, "qcons": None, "rcons": None,
            "score": best.double()}
