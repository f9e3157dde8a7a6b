"""Read search over the path cover (the automatic kernel of an index with its
k-mer table): equal to the oracle on the graphs and reads where runs end."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import sbwt_b200 as S
import sbwt_tools as T
from helpers import TMP, mixed_reads, oracle_index, oracle_results

pytestmark = pytest.mark.gpu


def genomes_of(kind: str, k: int) -> T.Genomes:
    if kind == "strains":  # branches every few k-mers
        return T.gen_genomes(5, 12, 4000, 2, 0.03, 0.03, 0.0)
    rng = np.random.default_rng(9)
    base = np.frombuffer(b"ACGT", np.uint8)
    if kind == "circular":  # one long cycle (each sequence repeats its first k - 1 chars)
        seqs = [base[rng.integers(0, 4, 3000)]]
        seqs = [np.concatenate([s, s[:k - 1]]) for s in seqs]
    else:  # short cycles: tandem repeats of 1 to 90 chars
        seqs = [np.tile(base[rng.integers(0, 4, u)], 1 + 200 // u) for u in (1, 2, 7, 40, 90)]
    return T.Genomes(np.concatenate(seqs), np.array([len(s) for s in seqs], np.uint64))


@pytest.mark.parametrize("kind", ["strains", "circular", "tandem"])
@pytest.mark.parametrize("k", [31, 30, 21, 13, 6])
def test_path_cover_matches_oracle(kind, k):
    import torch
    g = genomes_of(kind, k)
    path = TMP / f"cover_{kind}_{k}.sbwt"
    T.build_sbwt(g, k, str(path))
    idx = S.SbwtIndex.open(path)
    oracle = oracle_index(str(path), min(k, 6))
    src = g if kind != "tandem" else T.Genomes(np.concatenate([g.chars, g.chars, g.chars]),
                                               np.array([3 * len(g.chars)], np.uint64))
    for sub, n_rate in ((0.0, 0.0), (0.01, 0.005), (0.1, 0.03)):
        chars, ends = mixed_reads(src, 17, 700, median=90, sigma=0.8, sub=sub, n_rate=n_rate,
                                  frac=0.8, len_min=0, len_max=500)
        exp = oracle_results(oracle, chars, ends)
        d_chars = torch.from_numpy(chars.copy()).cuda()
        d_ends = torch.from_numpy(ends.view(np.int64).copy()).cuda()
        try:
            for tile in (0, 1, 31, 32, 33, 129):
                S.set_launch_config(tile=tile)
                out = torch.full((len(exp) + 4,), -7, dtype=torch.int64, device="cuda")
                assert idx.search_reads(d_chars, d_ends, out=out) == len(exp)
                got = out.cpu().numpy()
                assert np.array_equal(got[:len(exp)].view(np.uint64), exp)
                assert (got[len(exp):] == -7).all()
        finally:
            S.set_launch_config()
        assert np.array_equal(idx.search_reads(chars, ends), exp)  # 32-bit codes, widened


@pytest.mark.parametrize("kind", ["strains", "circular", "tandem"])
@pytest.mark.parametrize("k", [31, 21, 6])
def test_positions_over_the_cover_match_oracle(kind, k):
    """The positions seam with its k-mer table: stretches of consecutive
    positions of every length, steps back, repeats and scattered positions, up
    to the last k-mer of bit_seqs; one past it is an error."""
    import torch
    g = genomes_of(kind, k)
    path = TMP / f"cover_{kind}_{k}.sbwt"
    T.build_sbwt(g, k, str(path))
    idx = S.SbwtIndex.open(path)
    chars, ends = mixed_reads(g, 19, 200, median=60, sigma=0.5, sub=0.01, n_rate=0.01, frac=0.9,
                              len_min=0, len_max=200)
    chars = np.concatenate([chars, g.chars])[:len(chars) + (-len(chars)) % 32 + 32 * 4]
    bits, _ = O.seq_to_bits(chars.tobytes())
    bits = bits[:len(chars) // 32]  # no word past the last char
    last = len(chars) - k
    rng = np.random.default_rng(k)
    parts = [np.arange(last + 1), np.arange(last, -1, -1), rng.integers(0, last + 1, 500),
             np.full(40, last), np.arange(last - 40, last + 1)]
    for n in range(1, 70):
        a = int(rng.integers(0, last + 1 - n))
        parts.append(np.arange(a, a + n))
    pos = np.concatenate(parts).astype(np.uint64)
    exp = oracle_index(str(path), min(k, 6)).search_positions(bits, pos)
    assert np.array_equal(idx.search(bits, pos), exp)
    d_bits, d_pos = (torch.from_numpy(x.view(np.int64).copy()).cuda() for x in (bits, pos))
    for table in (True, False):
        idx.set_kmer_table(table)
        out = torch.full((len(pos) + 1,), -7, dtype=torch.int64, device="cuda")
        idx.search(d_bits, d_pos, out=out)
        got = out.cpu().numpy()
        assert np.array_equal(got[:-1].view(np.uint64), exp) and got[-1] == -7
    idx.set_kmer_table(True)
    with pytest.raises(S.SbwtError) as e:
        idx.search(bits, np.array([0, last + 1], np.uint64))
    assert e.value.code == S.E_INVALID


@pytest.mark.parametrize("k", [2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 29])
def test_labels_of_every_k(k):
    """The table's labels are put together by doublings and single steps chosen
    by the bits of k - 1: every k-mer of the index, and 2 000 others, found by
    the table as by the oracle."""
    g = genomes_of("strains", k)
    path = TMP / f"cover_labels_{k}.sbwt"
    T.build_sbwt(g, k, str(path))
    idx = S.SbwtIndex.open(path)
    rng = np.random.default_rng(k)
    noise = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 2000)]
    chars = np.concatenate([g.chars, noise])
    chars = chars[:len(chars) // 32 * 32]
    bits, _ = O.seq_to_bits(chars.tobytes())
    bits = bits[:len(chars) // 32]
    pos = np.arange(len(chars) - k + 1, dtype=np.uint64)
    exp = oracle_index(str(path), min(k, 6)).search_positions(bits, pos)
    assert np.array_equal(idx.search(bits, pos), exp)


def test_pipeline_batches_around_a_scan_block():
    """One pipeline, its graph updated from batch to batch: none, one, 1024 (a
    scan block), 1025 and more reads, in and out of order."""
    g = genomes_of("strains", 31)
    path = TMP / "cover_pipeline.sbwt"
    T.build_sbwt(g, 31, str(path))
    idx = S.SbwtIndex.open(path)
    chars, ends = mixed_reads(g, 23, 3000, median=90, sigma=0.6, sub=0.01, n_rate=0.01, frac=0.9,
                              len_min=0, len_max=400)
    pipe = S.Pipeline(idx, None, len(chars), len(ends))
    exp = oracle_results(oracle_index(str(path), 6), chars, ends)
    for n in (3000, 1, 1024, 1025, 0, 2048, 2049, 1, 1023, 3000):
        last = int(ends[n - 1]) if n else 0
        k = idx.count_kmers(ends[:n])
        assert np.array_equal(pipe.run(chars[:last], ends[:n]), exp[:k])
    pipe.close()


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 24, 29])
def test_reads_of_every_k(k):
    """From graphs that hold every k-mer to ones where a run is long, over the
    lines between the kernels and the lengths of the filter's L-mers."""
    import torch
    g = genomes_of("strains", k)
    path = TMP / f"cover_reads_{k}.sbwt"
    T.build_sbwt(g, k, str(path))
    idx = S.SbwtIndex.open(path)
    oracle = oracle_index(str(path), min(k, 6))
    for sub, n_rate, frac in ((0.0, 0.0, 1.0), (0.02, 0.005, 0.7), (0.2, 0.03, 0.5)):
        chars, ends = mixed_reads(g, 29, 600, median=90, sigma=0.8, sub=sub, n_rate=n_rate,
                                  frac=frac, len_min=0, len_max=500)
        exp = oracle_results(oracle, chars, ends)
        d_chars = torch.from_numpy(chars.copy()).cuda()
        d_ends = torch.from_numpy(ends.view(np.int64).copy()).cuda()
        out = torch.full((len(exp) + 4,), -7, dtype=torch.int64, device="cuda")
        assert idx.search_reads(d_chars, d_ends, out=out) == len(exp)
        got = out.cpu().numpy()
        assert np.array_equal(got[:len(exp)].view(np.uint64), exp)
        assert (got[len(exp):] == -7).all()
        assert np.array_equal(idx.search_reads(chars, ends), exp)
        n = C.c_uint64()
        out.fill_(-7)
        S.check(S.lib().sbwt_search_reads_noalloc(
            idx._h, d_chars.data_ptr(), d_chars.numel(), d_ends.data_ptr(), d_ends.numel(),
            out.data_ptr(), out.numel(), C.byref(n), 0, None))
        got = out.cpu().numpy()
        assert n.value == len(exp) and np.array_equal(got[:len(exp)].view(np.uint64), exp)
        assert (got[len(exp):] == -7).all()
        pipe = S.Pipeline(idx, None, len(chars), len(ends))
        for m in (600, 3, 600):
            last = int(ends[m - 1])
            assert np.array_equal(pipe.run(chars[:last], ends[:m]), exp[:idx.count_kmers(ends[:m])])
        pipe.close()


@pytest.mark.parametrize("k", [12, 13, 14, 15])
def test_short_k_with_a_large_table(k):
    """A table past the k-mers kernel's limit and 4^k from 2 to 130 times the
    k-mers: the automatic kernel equals the general one and the table kernel."""
    import torch
    rng = np.random.default_rng(31)
    chars = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 4_150_000)]
    path = TMP / f"cover_large_{k}.sbwt"
    S.build_index((chars, np.array([len(chars)], np.uint64)), k, path)
    idx = S.SbwtIndex.open(path)
    assert idx.set_kmer_table(True) + idx.filter_bytes() > 256 << 20
    reads = chars[:600_000].copy()
    for a, rate in ((150_000, 0.01), (300_000, 0.1), (450_000, 0.75)):
        hit = np.flatnonzero(rng.random(150_000) < rate) + a
        reads[hit] = np.frombuffer(b"ACGTN", np.uint8)[rng.choice(5, len(hit), p=[.24] * 4 + [.04])]
    ends = np.sort(rng.choice(np.arange(1, len(reads)), 5000, replace=False))
    d_reads = torch.from_numpy(reads).cuda()
    d_ends = torch.from_numpy(np.append(ends, len(reads)).astype(np.int64)).cuda()
    got = []
    try:
        for mode in (-1, 0, 1):
            S.set_table_kernel(mode)
            out = torch.full((len(reads) + 1,), -7, dtype=torch.int64, device="cuda")
            n = idx.search_reads(d_reads, d_ends, out=out)
            got.append(out.cpu().numpy())
            assert (got[-1][n:] == -7).all()
    finally:
        S.set_table_kernel()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("k", [5, 12, 13, 14])
@pytest.mark.parametrize("depth", [1, 2, 3, 4, 11, 12, 13, 14])
def test_positions_of_every_presearch_depth(k, depth):
    """The positions seam by presearch and steps or by the table, as k and the
    presearch depth decide."""
    if depth > k:
        pytest.skip("deeper than k")
    g = genomes_of("strains", k)
    path = TMP / f"cover_depth_{k}.sbwt"
    T.build_sbwt(g, k, str(path))
    idx = S.SbwtIndex.open(path, presearch_letters=depth)
    chars = g.chars[:len(g.chars) // 32 * 32].copy()
    rng = np.random.default_rng(depth)
    hit = rng.random(len(chars)) < 0.03
    chars[hit] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(hit.sum()))]
    bits, _ = O.seq_to_bits(chars.tobytes())
    bits = bits[:len(chars) // 32]
    pos = np.arange(len(chars) - k + 1, dtype=np.uint64)
    pos = np.concatenate([pos, rng.permutation(pos)])
    exp = oracle_index(str(path), min(k, 6)).search_positions(bits, pos)
    assert np.array_equal(idx.search(bits, pos), exp)
