"""Workloads whose speed this repository tracks, through its public entry points.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (an index built from seeded genomes and opened on the GPU,
reads, output buffers), ``run`` makes one pass through the binding or the C
ABI, ``work`` says which bytes a pass cannot do without.

All results are whole numbers (SBWT indexes, color ids, counts, text bytes),
so there is no rounding to compare: equal inputs give equal bytes.

Genomes and reads are seeded synthetic data, made on the GPU: genomes are
copies of random founders with substitutions (related strains), reads are
sampled from either strand of them with substitutions and Ns.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "sbwt-search_b200"))

import sbwt_b200 as S  # noqa: E402

DEV = "cuda:0"
TAU = 0.7

# The indexes the cases search (genomes x length, founders, substitutions).
INDEXES = {
    # one random 1 Mbp genome: tables that stay in L2
    "1mbp": dict(genomes=1, length=1_000_000, founders=0, sub=0.0),
    # ten strains of two species, 10 Mbp
    "10mbp": dict(genomes=10, length=1_000_000, founders=2, sub=0.02),
    # 40 strains of four species, 2.5 Mbp each: the headline index
    "100mbp": dict(genomes=40, length=2_500_000, founders=4, sub=0.02),
    # color indexes: many strains of eight species, and a few strains of two
    "2000strains": dict(genomes=2000, length=10_000, founders=8, sub=0.03),
    "100strains": dict(genomes=100, length=50_000, founders=2, sub=0.02),
}


def listed():
    return [
        # Interactive lookup of a few reads in a small index: call latency.
        dict(name="reads_100_small_index", kind="reads", index="1mbp", k=31, reads=100,
             median=150, sigma=0.0, sub=0.01, n_rate=0.0, random=0.5),
        # The CPU-comparable configuration: 100,000 reads, half of them foreign.
        dict(name="reads_100k_small_index", kind="reads", index="1mbp", k=31, reads=100_000,
             median=150, sigma=0.0, sub=0.01, n_rate=0.0, random=0.5),
        # The headline: a sequencing run against a 100 Mbp index, ragged lengths.
        dict(name="reads_3m_large_index", kind="reads", index="100mbp", k=31, reads=3_000_000,
             median=150, sigma=0.5, sub=0.005, n_rate=0.001, random=0.0),
        # Error-rich short reads (the batched workload's): mostly absent k-mers.
        dict(name="reads_2m_errors_large_index", kind="reads", index="100mbp", k=31,
             reads=2_000_000, median=100, sigma=0.0, sub=0.05, n_rate=0.0, random=0.0),
        # Long noisy reads, another k.
        dict(name="reads_long_k21", kind="reads", index="10mbp", k=21, reads=5_003,
             median=4_000, sigma=0.5, sub=0.05, n_rate=0.001, random=0.0),
        # The same call on host arrays, as a Python program makes it.
        dict(name="reads_host_200k", kind="reads_host", index="10mbp", k=31, reads=200_000,
             median=150, sigma=0.5, sub=0.005, n_rate=0.001, random=0.0),
        # The reference's own seam: packed chars and k-mer positions.
        dict(name="positions_4m", kind="positions", index="10mbp", k=31, reads=33_334,
             median=150, sigma=0.0, sub=0.01, n_rate=0.0, random=0.1),
        # Pseudoalignment of a batch of reads against 2000 strains.
        dict(name="pseudoalign_1m_2000_colors", kind="pseudoalign", index="2000strains", k=31,
             reads=1_000_000, median=150, sigma=0.0, sub=0.005, n_rate=0.0, random=0.0),
        # The reference's color seam: a count per read and color.
        dict(name="color_counts_20k", kind="counts", index="2000strains", k=31, reads=20_000,
             median=150, sigma=0.0, sub=0.005, n_rate=0.0, random=0.0),
        # Reads in, color ids out, on host memory: what a service runs per batch.
        dict(name="pipeline_20k", kind="pipeline", index="100strains", k=31, reads=20_000,
             median=150, sigma=0.0, sub=0.005, n_rate=0.0, random=0.05),
        # A FASTQ file's text to chars and read ends.
        dict(name="parse_fastq_1m", kind="parse", form="fastq", reads=1_000_000, median=150,
             sigma=0.5, wrap=0),
        # Index results of a batch to the reference's ascii lines.
        dict(name="format_index_ascii_1m", kind="format_index", fmt=0, k=31, reads=1_000_000,
             median=150, sigma=0.5, nodes=115_000_000, found=0.8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _reads(rng, most_chars, most_reads):
    """Read count, median length, spread and error rates of one drawn batch."""
    median = _log(rng, 50, 8_000)
    sigma = rng.choice([0.0, 0.0, 0.3, 0.5])
    hi = max(2, min(most_reads, int(most_chars / (median * math.exp(sigma * sigma / 2)))))
    return dict(reads=_log(rng, min(50, hi), hi), median=median, sigma=sigma,
                sub=rng.choice([0.0, 0.005, 0.01, 0.05]), n_rate=rng.choice([0.0, 0.0, 0.001]),
                random=rng.choice([0.0, 0.0, 0.1, 0.5]))


def draw(rng):
    kind = rng.choice(["reads", "reads", "reads", "reads", "reads_noalloc", "reads_host",
                       "positions", "pseudoalign", "pseudoalign", "counts", "pipeline",
                       "parse", "format_index", "format_colors"])
    if kind == "reads":
        c = dict(kind=kind, index=rng.choice(["1mbp", "10mbp", "100mbp"]), **_reads(rng, 400e6, 3_000_000))
        return dict(c, k=rng.choice([31, 31, 31, 27, 21, 16]))
    if kind == "reads_noalloc":  # at most 8 Mi chars and 256 Ki reads per call
        c = dict(kind=kind, index=rng.choice(["1mbp", "10mbp"]), **_reads(rng, 5e6, 200_000))
        return dict(c, k=rng.choice([31, 21]))
    if kind == "reads_host":
        c = dict(kind=kind, index=rng.choice(["1mbp", "10mbp"]), **_reads(rng, 40e6, 300_000))
        return dict(c, k=rng.choice([31, 25]))
    if kind == "positions":
        c = dict(kind=kind, index=rng.choice(["1mbp", "10mbp"]), **_reads(rng, 10e6, 100_000))
        return dict(c, n_rate=0.0, k=rng.choice([31, 23]))
    if kind in ("pseudoalign", "counts", "pipeline"):
        most = {"pseudoalign": 400_000, "counts": 20_000, "pipeline": 30_000}[kind]
        c = dict(kind=kind, index=rng.choice(["2000strains", "100strains"]),
                 **_reads(rng, most * 150, most))
        return dict(c, k=31, median=min(c["median"], 2_000))
    if kind == "parse":
        form = rng.choice(["fastq", "fasta"])
        c = _reads(rng, 150e6, 1_000_000)
        return dict(kind=kind, form=form, reads=c["reads"], median=c["median"], sigma=c["sigma"],
                    wrap=rng.choice([60, 80]) if form == "fasta" else 0)
    if kind == "format_index":
        c = _reads(rng, 150e6, 1_000_000)
        return dict(kind=kind, fmt=rng.choice([0, 0, 1, 2]), k=31, reads=c["reads"],
                    median=c["median"], sigma=c["sigma"], nodes=_log(rng, 100_000, 1_000_000_000),
                    found=rng.choice([0.2, 0.8, 1.0]))
    fmt = rng.choice([0, 0, 1, 2])
    return dict(kind=kind, fmt=fmt, colors=_log(rng, 16, 3_000),
                reads=_log(rng, 100, 30_000 if fmt == 2 else 2_000_000),
                per_read=rng.choice([2, 10, 40]))


# -- inputs ------------------------------------------------------------------

ASCII = (65, 67, 71, 84)  # A C G T


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1_000_003 + salt)


def _ascii(codes):
    return torch.tensor(ASCII, dtype=torch.uint8, device=DEV)[codes.long()]


def _mutate(codes, rate, g):
    if rate:
        hit = torch.rand(codes.shape, device=DEV, generator=g) < rate
        add = torch.randint(1, 4, codes.shape, device=DEV, dtype=torch.uint8, generator=g)
        codes = torch.where(hit, (codes + add) & 3, codes)
    return codes


def _genomes(index, seed):
    """(genomes, length) 2-bit codes."""
    ix, g = INDEXES[index], _gen(seed, 1)
    n, length, f = ix["genomes"], ix["length"], ix["founders"]
    codes = torch.randint(0, 4, (f or n, length), device=DEV, dtype=torch.uint8, generator=g)
    return _mutate(codes[torch.arange(n, device=DEV) % f], ix["sub"], g) if f else codes


def _lengths(case, g, hi):
    """Log-normal read lengths: its quantiles in an order of the seed's (so a
    case has as many chars and k-mers with every seed)."""
    n, median = case["reads"], float(case["median"])
    q = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n
    z = torch.erfinv(2 * q - 1) * math.sqrt(2) * case["sigma"]
    lens = (torch.exp(z) * median).round().long()
    lens = lens.clamp(min(31, int(median)), int(min(hi, median * 7)))
    return lens[torch.randperm(n, device=DEV, generator=g)]


def _ragged(starts, lens):
    """Index of every char of ragged spans [starts, starts + lens), and each char's span."""
    ends = torch.cumsum(lens, 0)
    total = int(ends[-1])
    span = torch.repeat_interleave(torch.arange(len(lens), device=DEV), lens, output_size=total)
    inside = torch.arange(total, device=DEV) - (ends - lens)[span]
    return starts[span] + inside, span, inside, ends


def _sample_reads(case, genomes, seed):
    """Reads from random places and strands: (ascii chars, cumulative ends)."""
    g = _gen(seed, 2)
    n, length = genomes.shape
    lens = _lengths(case, g, length)
    at = torch.randint(0, n, (len(lens),), device=DEV, generator=g) * length
    at += (torch.rand(len(lens), device=DEV, generator=g, dtype=torch.float64) *
           (length - lens + 1)).long()
    back = torch.rand(len(lens), device=DEV, generator=g) < 0.5
    pos, span, inside, ends = _ragged(at, lens)
    flip = back[span]
    pos = torch.where(flip, at[span] + lens[span] - 1 - inside, pos)
    codes = genomes.reshape(-1)[pos]
    codes = torch.where(flip, 3 - codes, codes)
    codes = _mutate(codes, case["sub"], g)
    if case["random"]:
        foreign = (torch.rand(len(lens), device=DEV, generator=g) < case["random"])[span]
        other = torch.randint(0, 4, codes.shape, device=DEV, dtype=torch.uint8, generator=g)
        codes = torch.where(foreign, other, codes)
    chars = _ascii(codes)
    if case["n_rate"]:
        unknown = torch.rand(chars.shape, device=DEV, generator=g) < case["n_rate"]
        chars = torch.where(unknown, torch.full_like(chars, 78), chars)
    return chars, ends


def _open_index(case, genomes):
    n, length = genomes.shape
    chars = _ascii(genomes.reshape(-1)).cpu().numpy()
    ends = np.arange(1, n + 1, dtype=np.uint64) * np.uint64(length)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "index.sbwt")
        S.build_index((chars, ends), case["k"], path)
        return S.SbwtIndex.open(path)


def _open_colored(case, genomes):
    n, length = genomes.shape
    chars = _ascii(genomes.reshape(-1)).cpu().numpy()
    ends = np.arange(1, n + 1, dtype=np.uint64) * np.uint64(length)
    with tempfile.TemporaryDirectory() as d:
        sbwt, colors = os.path.join(d, "index.sbwt"), os.path.join(d, "index.tcolors")
        S.build_colored_index(chars, ends, case["k"], sbwt, colors)
        return S.SbwtIndex.open(sbwt), S.ColorIndex.open(colors)


def _kmers(ends, k):
    lens = torch.diff(ends, prepend=torch.zeros(1, dtype=ends.dtype, device=DEV))
    return (lens - k + 1).clamp(min=0)


def _results_buffer(ends, k):
    return torch.empty(max(1, int(_kmers(ends, k).sum())), dtype=torch.int64, device=DEV)


def _found(index, chars, ends, k):
    """Found SBWT indexes of every read and their offsets: the colors step's input."""
    out = _results_buffer(ends, k)
    per = _kmers(ends, k)
    n = index.search_reads(chars, ends, out=out)
    read = torch.repeat_interleave(torch.arange(len(per), device=DEV), per, output_size=n)
    hit = out[:n] >= 0
    counts = torch.bincount(read[hit], minlength=len(per))
    offs = torch.zeros(len(per) + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(counts, 0, out=offs[1:])
    return out[:n][hit].contiguous(), offs


def _text(case, seed):
    """FASTQ or line-wrapped FASTA text of random reads (uint8, on the GPU)."""
    g = _gen(seed, 3)
    lens = _lengths(case, g, 100_000)
    wrap = case["wrap"]
    if case["form"] == "fastq":
        tail = lens + 4  # "\n+\n", qualities, "\n"
        body = lens
    else:
        body = lens + (lens + wrap - 1) // wrap  # a newline after every line
        tail = torch.zeros_like(lens)
    head = 2 + torch.arange(len(lens), device=DEV) % 7  # name chars
    rec = 1 + head + 1 + body + tail
    start = torch.cumsum(rec, 0) - rec
    text = torch.full((int(rec.sum()),), 73, dtype=torch.uint8, device=DEV)  # 'I'
    text[start] = 64 if case["form"] == "fastq" else 62
    seq = start + 1 + head
    text[seq] = 10
    seq = seq + 1
    pos, span, inside, _ = _ragged(seq, lens)
    if wrap:
        pos = pos + inside // wrap
    text[pos] = _ascii(torch.randint(0, 4, pos.shape, device=DEV, dtype=torch.uint8, generator=g))
    if wrap:
        last = (inside % wrap == wrap - 1) | (inside == lens[span] - 1)
        text[pos[last] + 1] = 10
    else:
        text[seq + lens] = 10
        text[seq + lens + 1] = 43
        text[seq + lens + 2] = 10
        text[start + rec - 1] = 10
    return text, int(lens.sum())


# -- cases -------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind in ("reads", "reads_noalloc", "reads_host", "positions"):
        genomes = _genomes(case["index"], seed)
        st["index"] = _open_index(case, genomes)
        chars, ends = _sample_reads(case, genomes, seed)
        if kind == "reads_host":
            st["chars"], st["ends"] = chars.cpu().numpy(), ends.cpu().numpy().view(np.uint64)
        elif kind == "positions":
            codes = ((chars >> 1) ^ (chars >> 2)).long() & 3
            codes = torch.nn.functional.pad(codes, (0, 64 - len(codes) % 32)).view(-1, 32)
            shift = 62 - 2 * torch.arange(32, device=DEV)
            st["bits"] = (codes << shift).sum(1)
            per = _kmers(ends, case["k"])
            lens = torch.diff(ends, prepend=torch.zeros(1, dtype=ends.dtype, device=DEV))
            st["positions"] = _ragged(ends - lens, per)[0].contiguous()
            st["out"] = torch.empty_like(st["positions"])
        else:
            st["chars"], st["ends"] = chars, ends
            st["out"] = _results_buffer(ends, case["k"])
    elif kind in ("pseudoalign", "counts", "pipeline"):
        genomes = _genomes(case["index"], seed)
        st["index"], st["colors"] = _open_colored(case, genomes)
        chars, ends = _sample_reads(case, genomes, seed)
        if kind == "pipeline":
            st["chars"], st["ends"] = chars.cpu().numpy(), ends.cpu().numpy().view(np.uint64)
            st["pipeline"] = S.Pipeline(st["index"], st["colors"], len(chars), len(ends), tau=TAU)
            st["ids"] = np.zeros(len(ends) * 64 + 4096, dtype=np.uint32)
            st["ids_offs"] = np.zeros(len(ends) + 1, dtype=np.uint64)
        else:
            st["found"], st["offs"] = _found(st["index"], chars, ends, case["k"])
            n = len(ends)
            if kind == "counts":
                st["counts"] = torch.empty((n, st["colors"].num_colors), dtype=torch.int32,
                                           device=DEV)
            else:
                st["ids_offs"] = torch.empty(n + 1, dtype=torch.int64, device=DEV)
                st["ids"] = torch.zeros(n * 64 + 4096, dtype=torch.int32, device=DEV)
    elif kind == "parse":
        st["text"], chars = _text(case, seed)
        st["chars"] = torch.empty(max(1, chars), dtype=torch.uint8, device=DEV)
        st["ends"] = torch.empty(case["reads"], dtype=torch.int64, device=DEV)
    elif kind == "format_index":
        g = _gen(seed, 4)
        st["ends"] = torch.cumsum(_lengths(case, g, 100_000), 0)
        n = int(_kmers(st["ends"], case["k"]).sum())
        res = torch.randint(0, case["nodes"], (n,), device=DEV, generator=g)
        miss = torch.rand(n, device=DEV, generator=g) >= case["found"]
        st["results"] = torch.where(miss, torch.full_like(res, -1), res)
        st["out"] = torch.zeros({0: 11 * n, 1: 8 * n, 2: n}[case["fmt"]] + 8 * case["reads"],
                                dtype=torch.uint8, device=DEV)
    else:
        g = _gen(seed, 5)
        per = torch.arange(case["reads"], device=DEV) % (2 * case["per_read"] + 1)
        per = per.clamp(max=case["colors"])[torch.randperm(len(per), device=DEV, generator=g)]
        st["offs"] = torch.zeros(case["reads"] + 1, dtype=torch.int64, device=DEV)
        torch.cumsum(per, 0, out=st["offs"][1:])
        n = int(st["offs"][-1])
        read = torch.repeat_interleave(torch.arange(case["reads"], device=DEV), per, output_size=n)
        inside = torch.arange(n, device=DEV) - st["offs"][read]
        st["ids"] = (inside * case["colors"] // per[read]).to(torch.int32)  # ascending, distinct
        shift = torch.randint(0, case["colors"], (case["reads"],), device=DEV, generator=g)
        st["ids"] = torch.sort((read << 32) + (st["ids"] + shift[read]) % case["colors"])[0]
        st["ids"] = (st["ids"] & 0xFFFFFFFF).to(torch.int32)
        size = {0: 5 * n, 1: 8 * n, 2: 2 * case["colors"] * case["reads"]}[case["fmt"]]
        st["out"] = torch.zeros(size + 8 * case["reads"], dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()  # the parser and the formatters run on a stream of their own
    return st


def run(st):
    """One pass.  Buffers whose filled part depends on the data (color ids,
    formatted text) are the caller's, zeroed once, and come back whole."""
    kind = st["kind"]
    if kind == "reads":
        n = st["index"].search_reads(st["chars"], st["ends"], out=st["out"])
        return st["out"][:n]
    if kind == "reads_noalloc":
        n, out = C.c_uint64(), st["out"]
        S.check(S.lib().sbwt_search_reads_noalloc(
            st["index"]._h, C.c_void_p(st["chars"].data_ptr()), C.c_uint64(len(st["chars"])),
            C.c_void_p(st["ends"].data_ptr()), C.c_uint64(len(st["ends"])),
            C.c_void_p(out.data_ptr()), C.c_uint64(len(out)), C.byref(n), C.c_uint32(0), None))
        return out[:n.value]
    if kind == "reads_host":
        return st["index"].search_reads(st["chars"], st["ends"]).view(np.int64)
    if kind == "positions":
        return st["index"].search(st["bits"], st["positions"], out=st["out"])
    if kind == "pseudoalign":
        n, offs = len(st["offs"]) - 1, st["ids_offs"]
        S.check(S.lib().sbwt_pseudoalign(
            st["colors"]._h, st["found"].data_ptr(), st["offs"].data_ptr(), None, None, n, TAU,
            S.DEVICE_POINTERS, st["ids"].data_ptr(), len(st["ids"]), offs.data_ptr(), None))
        return st["ids"], offs
    if kind == "counts":
        S.check(S.lib().sbwt_color_counts(
            st["colors"]._h, st["found"].data_ptr(), st["offs"].data_ptr(), len(st["offs"]) - 1,
            st["counts"].data_ptr(), S.DEVICE_POINTERS, None))
        return st["counts"]
    if kind == "pipeline":
        chars, ends, n = st["chars"], st["ends"], C.c_uint64()
        ids, offs = st["ids"], st["ids_offs"]
        S.check(S.lib().sbwt_pipeline_run(
            st["pipeline"]._h, chars.ctypes.data, len(chars), ends.ctypes.data, len(ends), None, 0,
            C.byref(n), ids.ctypes.data, len(ids), offs.ctypes.data))
        return ids.view(np.int32), offs.view(np.int64)
    if kind == "parse":
        text, chars, ends = st["text"], st["chars"], st["ends"]
        nc, nr = C.c_uint64(), C.c_uint64()
        S.check(S.lib().sbwt_fastx_parse(
            text.data_ptr(), len(text), chars.data_ptr(), len(chars), ends.data_ptr(), len(ends),
            C.byref(nc), C.byref(nr), S.DEVICE_POINTERS, 0, None))
        return chars[:nc.value], ends[:nr.value]
    size, out = C.c_uint64(), st["out"]
    case = st["case"]
    if kind == "format_index":
        S.check(S.lib().sbwt_format_index_results(
            st["results"].data_ptr(), st["ends"].data_ptr(), len(st["ends"]), case["k"],
            case["fmt"], out.data_ptr(), len(out), C.byref(size), S.DEVICE_POINTERS, 0, None))
    else:
        S.check(S.lib().sbwt_format_color_results(
            st["ids"].data_ptr(), st["offs"].data_ptr(), len(st["offs"]) - 1, case["colors"],
            case["fmt"], out.data_ptr(), len(out), C.byref(size), S.DEVICE_POINTERS, 0, None))
    return out, size.value


def work(case):
    """Input and output bytes of a pass, each moved once; the index's own
    tables, of which a pass reads what its k-mers hit, are left out."""
    kind, n = case["kind"], case["reads"]
    if kind == "format_colors":
        ids = n * min(case["per_read"], case["colors"])
        out = {0: ids * 4 + n, 1: 8 * (ids + n), 2: 2 * n * case["colors"]}[case["fmt"]]
        return {"bytes": 4 * ids + 8 * n + out, "flops": 0}
    mean = case["median"] * math.exp(case["sigma"] ** 2 / 2)
    chars = n * mean
    if kind == "parse":
        text = 2 * chars + 8 * n if case["form"] == "fastq" else chars * (1 + 1 / case["wrap"])
        return {"bytes": text + chars + 8 * n, "flops": 0}
    kmers = n * max(1.0, mean - case["k"] + 1)
    if kind == "format_index":
        width = case["found"] * (math.log10(case["nodes"]) + 1) + (1 - case["found"]) * 3
        out = {0: width * kmers, 1: 8 * (kmers + n), 2: kmers + n}[case["fmt"]]
        return {"bytes": 8 * kmers + 8 * n + out, "flops": 0}
    if kind == "positions":
        return {"bytes": chars / 4 + 16 * kmers, "flops": 0}
    if kind == "counts":
        return {"bytes": 8 * kmers + 8 * n + 4 * n * INDEXES[case["index"]]["genomes"], "flops": 0}
    if kind == "pseudoalign":
        return {"bytes": 8 * kmers + 16 * n + 4 * n, "flops": 0}
    if kind == "pipeline":
        return {"bytes": chars + 16 * n + 4 * n, "flops": 0}
    return {"bytes": chars + 8 * n + 8 * kmers, "flops": 0}
