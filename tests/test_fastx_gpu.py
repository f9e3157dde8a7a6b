"""FASTA/FASTQ parsing on the GPU (sbwt_fastx_parse) against the host reader
(sbwt_fastx_read, pinned to the reference's fixtures): identical chars and
read ends on the fixtures, on seeded adversarial text and on layouts that put
1024-line chunk boundaries inside sequences and qualities."""
import ctypes as C

import numpy as np
import pytest

import sbwt_b200 as S
from helpers import FIXTURE_FILES, GOLDEN, host_fastx, random_fastx

pytestmark = pytest.mark.gpu


def check_same(text, tmp_path):
    hc, he = host_fastx(text, tmp_path / "in.fx")
    dc, de = S.fastx_parse(text)
    assert dc.tobytes() == hc
    assert de.tolist() == he.tolist()
    return len(he)


@pytest.mark.parametrize("name", FIXTURE_FILES)
def test_fixtures(name, tmp_path):
    check_same((GOLDEN / "index_search" / name).read_bytes(), tmp_path)


@pytest.mark.parametrize("seed", range(8))
def test_random_text(seed, tmp_path):
    # ~10-40 k lines: many chunks, boundaries anywhere in the records
    text = random_fastx(100 + seed, 4000, fastq_frac=[0.0, 0.5, 1.0, 0.8][seed % 4],
                        max_line=[80, 7, 200, 3][seed % 4], final_newline=seed % 3 != 0)
    assert check_same(text, tmp_path) > 0


def test_edge_cases(tmp_path):
    cases = [b"", b"\n", b">", b">\n", b"@\n", b"ACGT\n", b">a\nAC\r\nGT\r",
             b">a\r\nAC\r\nGT\n>b\n>c\nTT\n\n@q x\nACG\nT\n+\nII\nII\n@r\n\n+\n\n",
             b"@a\nACGT\n+\n@@\n", b"@a\nACGT\n+\n@@@@\n@b\nA\n+\n>\n",
             b"@a\nAC\n+\nII", b"\r\n\r\n>x\r\n\r\nA\r\n", b"+\n@a\n+\n+\n"]
    for t in cases:
        check_same(t, tmp_path)


def test_long_fasta_records_across_chunks(tmp_path):
    # 3 records of 6000 lines each: whole chunks inside one sequence
    rng = np.random.default_rng(7)
    parts = []
    for r in range(3):
        parts.append(b">chr%d\n" % r)
        body = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 60 * 6000))
        parts += [body[i:i + 60] + b"\n" for i in range(0, len(body), 60)]
    assert check_same(b"".join(parts), tmp_path) == 3


def test_fastq_shifted_by_a_junk_line(tmp_path):
    # 4-line records after one junk line: every chunk starts inside a record
    rng = np.random.default_rng(8)
    lines = [b"junk"]
    for r in range(3000):
        s = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 100))
        q = b"@" + bytes(rng.choice(np.frombuffer(b"I@+>", np.uint8), 99))
        lines += [b"@q%d" % r, s, b"+", q]
    assert check_same(b"\n".join(lines) + b"\n", tmp_path) == 3000


def test_device_pointers_and_capacity():
    import torch
    text = random_fastx(5, 500)
    hc, he = S.fastx_parse(text)
    d_text = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    d_chars = torch.zeros(len(text), dtype=torch.uint8, device="cuda")
    d_ends = torch.zeros(len(he), dtype=torch.int64, device="cuda")
    nc, nr = C.c_uint64(), C.c_uint64()
    L = S.lib()
    rc = L.sbwt_fastx_parse(d_text.data_ptr(), len(text), d_chars.data_ptr(), len(text),
                            d_ends.data_ptr(), len(he) - 1, C.byref(nc), C.byref(nr),
                            S.DEVICE_POINTERS, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == S.E_CAPACITY and nr.value == len(he) and nc.value == len(hc)
    S.check(L.sbwt_fastx_parse(d_text.data_ptr(), len(text), d_chars.data_ptr(), len(text),
                               d_ends.data_ptr(), len(he), C.byref(nc), C.byref(nr),
                               S.DEVICE_POINTERS, 0, torch.cuda.current_stream().cuda_stream))
    assert d_chars[:nc.value].cpu().numpy().tobytes() == hc.tobytes()
    assert d_ends.cpu().numpy().view(np.uint64).tolist() == he.tolist()


def _layout(kind: str, n: int) -> bytes:
    rng = np.random.default_rng(n)
    base = np.frombuffer(b"ACGTN", np.uint8)

    def seq(m):
        return bytes(rng.choice(base, m))

    if kind == "fastq":  # four lines a record: chunks start on records
        return b"".join(b"@r\n%s\n+\n%s\n" % (s, b"@" * len(s))
                        for s in (seq(int(rng.integers(1, 300))) for _ in range(n)))
    if kind == "one_char_lines":  # hundreds of lines in 512 output bytes
        return b">x\n" + b"".join(seq(1) + b"\n" for _ in range(n)) + b">y\r\n" + seq(n) + b"\r\n"
    if kind == "one_line":
        return b">x\n" + seq(n)
    return b"".join(b">%d\n%s\n\n" % (i, b"\r\n".join(seq(w) for w in (1, 15, 16, 17, i % 70 + 1)))
                    for i in range(n))


@pytest.mark.parametrize("kind", ["fastq", "one_char_lines", "one_line", "wrapped"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 700, 40_000])
def test_layouts_at_every_alignment(kind, n, tmp_path):
    """Texts and outputs at any place in a 16-byte line, lines from one char to
    the whole text, chunks entered searching and inside a sequence; nothing is
    written around the outputs."""
    import torch
    text = _layout(kind, n)
    hc, he = host_fastx(text, tmp_path / "in.fx")
    L, nc, nr = S.lib(), C.c_uint64(), C.c_uint64()
    for a, b in ((0, 0), (1, 15), (7, 8), (15, 1)):
        buf = np.full(a + len(text) + 16, ord("\n"), np.uint8)
        buf[a:a + len(text)] = np.frombuffer(text, np.uint8)
        d_text = torch.from_numpy(buf).cuda()
        d_chars = torch.full((b + len(hc) + 16,), 7, dtype=torch.uint8, device="cuda")
        d_ends = torch.full((len(he) + 1,), -7, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        S.check(L.sbwt_fastx_parse(d_text.data_ptr() + a, len(text), d_chars.data_ptr() + b,
                                   len(hc), d_ends.data_ptr(), len(he), C.byref(nc),
                                   C.byref(nr), S.DEVICE_POINTERS, 0, None))
        assert (nc.value, nr.value) == (len(hc), len(he))
        out = d_chars.cpu().numpy()
        assert out[b:b + len(hc)].tobytes() == hc
        assert (out[:b] == 7).all() and (out[b + len(hc):] == 7).all()
        ends = d_ends.cpu().numpy()
        assert ends[:-1].tolist() == he.tolist() and ends[-1] == -7


@pytest.mark.parametrize("lines", [*range(1, 20), 31, 32, 33, 39, 40, 41, 63, 64, 65, 8191, 8193])
@pytest.mark.parametrize("newline", [False, True])
def test_line_counts_around_the_groups(lines, newline, tmp_path):
    """Newline entries are read eight at a time, the last group's one by one:
    every number of lines in a group, with and without a newline at the end."""
    rng = np.random.default_rng(lines)
    rows = [b">%d" % i if i % 5 == 0 else b"ACGTN"[:int(rng.integers(0, 6))] for i in range(lines)]
    check_same(b"\n".join(rows) + (b"\n" if newline else b""), tmp_path)


def _records(n: int, shift: int, per: int, first: bytes) -> bytes:
    """n FASTQ records of `per` sequence and `per` quality lines after `shift`
    blank lines; every quality line starts with `first`."""
    rows = [b""] * shift
    for i in range(n):
        rows += [b"@r%d" % i, *[b"ACGT"] * per, b"+", *[first + b"II" + first] * per]
    return b"\n".join(rows) + b"\n"


@pytest.mark.parametrize("first", [b"@", b">", b"+", b"I"])
@pytest.mark.parametrize("per", [1, 2])
def test_last_group_entered_inside_a_sequence(per, first, tmp_path):
    """Lines are summed up in groups of 32.  A group that is entered inside a
    sequence and meets a '+' line first has no sum, the last group of a text
    included, which no other group follows: 33 to 96 lines at every shift of
    the records against the groups, from host and device pointers."""
    import torch
    L, nc, nr = S.lib(), C.c_uint64(), C.c_uint64()
    for shift in range(4):
        for n in range(32 // (2 + 2 * per), 96 // (2 + 2 * per) + 1):
            text = _records(n, shift, per, first)
            assert check_same(text, tmp_path) == n
            hc, he = host_fastx(text, tmp_path / "in.fx")
            d_text = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
            d_chars = torch.full((len(hc) + 1,), 7, dtype=torch.uint8, device="cuda")
            d_ends = torch.full((n + 1,), -7, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            S.check(L.sbwt_fastx_parse(d_text.data_ptr(), len(text), d_chars.data_ptr(), len(hc),
                                       d_ends.data_ptr(), n, C.byref(nc), C.byref(nr),
                                       S.DEVICE_POINTERS, 0, None))
            assert (nc.value, nr.value) == (len(hc), n)
            assert d_chars.cpu().numpy().tobytes() == hc + b"\x07"
            assert d_ends.cpu().numpy().tolist() == [*he.tolist(), -7]


@pytest.mark.parametrize("before", [14, 15, 16, 23_999, 39_999])
def test_fastq_record_after_fasta(before, tmp_path):
    """FASTA records, then one FASTQ record that may lie across the last group's
    start; the largest has more groups than one block sums up."""
    text = b"".join(b">%d\nAC\n" % i for i in range(before)) + b"@q\nACGT\n+\n@III\n"
    assert check_same(text, tmp_path) == before + 1


@pytest.mark.parametrize("first", [b"@", b">", b"+", b"I"])
@pytest.mark.parametrize("per", [1, 3, 4, 17, 40])
def test_fix_up_of_long_records(per, first, tmp_path):
    """Records of 4 to 82 lines, most of them entered inside by a group of 1024
    lines: the line on which its first guess and the truth meet lies among the
    group's first eight lines, in one of the runs of 32 after them, or nowhere."""
    n = 12_000 // (2 + 2 * per)
    for shift in (1, 2, 5):
        assert check_same(_records(n, shift, per, first), tmp_path) == n


@pytest.mark.parametrize("kind", ["fastq", "short lines", "long lines"])
@pytest.mark.parametrize("lead", [0, 5])
def test_large_text(kind, lead, tmp_path):
    """Texts past the sizes of one block's scan of the newline counts (33 MB) and
    of the copy's smallest range (9.7 M output chars): reads of 0 to 400 chars,
    10 M lines of one or two chars, and lines of up to 3 MB, with text and output
    on and off a 16-byte boundary."""
    import torch
    rng = np.random.default_rng(len(kind))
    seq = np.frombuffer(b"ACGTN", np.uint8)[rng.integers(0, 5, 4 << 20)].tobytes()
    if kind == "fastq":
        at, n = rng.integers(0, len(seq) - 400, 120_000), rng.integers(0, 401, 120_000)
        text = b"".join(b"@%d\n%s\n+\n%s\n" % (i, seq[a:a + m], b"I" * m)
                        for i, (a, m) in enumerate(zip(at, n)))
    elif kind == "short lines":
        lines = np.full((10_500_000, 3), ord("\n"), np.uint8)
        lines[:, 0] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, len(lines))]
        two = rng.random(len(lines)) < 0.3
        lines[two, 1] = ord("G")
        lines[rng.integers(0, len(lines), 1000), 0] = ord(">")
        keep = np.ones(lines.shape, bool)
        keep[~two, 2] = False
        text = b">x\n" + lines[keep].tobytes() + b">y\nA"
    else:
        text = b"".join(b">%d\n%s\n" % (i, seq[a:a + m]) for i, (a, m) in enumerate(
            zip(rng.integers(0, 1 << 20, 30), rng.integers(0, 3_000_000, 30))))
    assert len(text) > 22_000_000
    hc, he = host_fastx(text, tmp_path / "in.fx")
    assert len(hc) > 10_000_000
    d_text = torch.from_numpy(np.frombuffer(b"\n" * lead + text, np.uint8).copy()).cuda()
    d_chars = torch.full((lead + len(hc) + 16,), 7, dtype=torch.uint8, device="cuda")
    d_ends = torch.full((len(he) + 1,), -7, dtype=torch.int64, device="cuda")
    nc, nr = C.c_uint64(), C.c_uint64()
    torch.cuda.synchronize()
    S.check(S.lib().sbwt_fastx_parse(d_text.data_ptr() + lead, len(text),
                                     d_chars.data_ptr() + lead, len(hc), d_ends.data_ptr(),
                                     len(he), C.byref(nc), C.byref(nr), S.DEVICE_POINTERS, 0, None))
    assert (nc.value, nr.value) == (len(hc), len(he))
    h = d_chars.cpu().numpy()
    assert h[lead:lead + len(hc)].tobytes() == hc
    assert (h[:lead] == 7).all() and (h[lead + len(hc):] == 7).all()
    e = d_ends.cpu().numpy()
    assert np.array_equal(e[:-1].view(np.uint64), he) and e[-1] == -7
