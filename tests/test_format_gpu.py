"""Result formatting on the GPU (sbwt_format_index_results /
sbwt_format_color_results) against the host writers, which reproduce the
reference's files byte for byte: every format, adversarial values, empty
reads, the golden fixtures' expected ascii files, and device buffers."""
import ctypes as C
import struct

import numpy as np
import pytest

import oracle as O
import sbwt_b200 as S
from helpers import FIXTURE_FILES, GOLDEN, TMP, golden_sbwt_path, host_fastx, oracle_index

pytestmark = pytest.mark.gpu
EXT_INDEX = {0: ".txt", 1: ".bin", 2: ".bool"}
EXT_COLOR = {0: ".txt", 1: ".bin", 2: ".csv"}


def host_index_bytes(res, ends, k, fmt, name):
    L = S.lib()
    L.sbwt_write_index_results.argtypes = [C.c_char_p, C.c_int, C.c_int, C.c_void_p,
                                           C.c_void_p, C.c_uint64, C.c_uint32]
    out = TMP / name
    S.check(L.sbwt_write_index_results(str(out).encode(), fmt, 0,
                                       res.ctypes.data if len(res) else None,
                                       ends.ctypes.data if len(ends) else None, len(ends), k))
    return (TMP / (name + EXT_INDEX[fmt])).read_bytes()


def host_color_bytes(ids, offs, C_, fmt, name):
    L = S.lib()
    L.sbwt_write_color_results.argtypes = [C.c_char_p, C.c_int, C.c_int, C.c_void_p,
                                           C.c_void_p, C.c_uint64, C.c_uint64]
    out = TMP / name
    S.check(L.sbwt_write_color_results(str(out).encode(), fmt, 0,
                                       ids.ctypes.data if len(ids) else None, offs.ctypes.data,
                                       len(offs) - 1, C_))
    b = (TMP / (name + EXT_COLOR[fmt])).read_bytes()
    return b[b.index(b"\n") + 1:] if fmt == 2 else b  # csv: drop the title row


def random_index_batch(seed, n_reads, k=31):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 3 * k, n_reads)
    lens[rng.random(n_reads) < 0.1] = int(rng.integers(0, k))  # reads shorter than k
    ends = np.cumsum(lens).astype(np.uint64)
    nk = int(np.maximum(lens - k + 1, 0).sum())
    res = rng.integers(0, 1 << 40, nk, dtype=np.uint64)
    small = rng.random(nk) < 0.5
    res[small] = rng.integers(0, 1000, int(small.sum()), dtype=np.uint64)
    res[rng.random(nk) < 0.2] = O.NOT_FOUND
    res[rng.random(nk) < 0.1] = O.INVALID
    res[rng.random(nk) < 0.02] = np.uint64(O.INVALID - 1)  # 20-digit value
    return res, ends


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("seed", [1, 2])
def test_index_formats_match_host_writer(fmt, seed):
    res, ends = random_index_batch(seed, 3000 + seed)
    got = S.format_index_results(res, ends, 31, fmt)
    assert got == host_index_bytes(res, ends, 31, fmt, f"fi_{seed}_{fmt}")


@pytest.mark.parametrize("name", FIXTURE_FILES)
def test_index_ascii_reproduces_reference_fixture(name, tmp_path):
    idx = oracle_index(golden_sbwt_path(), 10)
    text = (GOLDEN / "index_search" / name).read_bytes()
    chars, ends = host_fastx(text, tmp_path / "q.fx")
    reads = O.parse_fastx(text)
    res = np.concatenate(O.index_search_reads(idx, reads) + [np.zeros(0, np.uint64)])
    body = S.format_index_results(res.astype(np.uint64), ends, 30, 0)
    head = b"".join(struct.pack("<Q", len(s)) + s for s in (b"ascii", b"v1.0"))
    exp = (GOLDEN / "index_search" / "expected" / (name.split(".")[0] + ".txt")).read_bytes()
    assert head + body == exp


@pytest.mark.parametrize("fmt", [0, 1, 2])
def test_color_formats_match_host_writer(fmt):
    rng = np.random.default_rng(fmt)
    n_reads, n_colors = 2500, 3000
    counts = rng.integers(0, 40, n_reads)
    counts[rng.random(n_reads) < 0.3] = 0
    offs = np.zeros(n_reads + 1, np.uint64)
    offs[1:] = np.cumsum(counts)
    ids = np.concatenate([np.sort(rng.choice(n_colors, int(c), replace=False))
                          for c in counts]).astype(np.uint32)
    got = S.format_color_results(ids, offs, n_colors, fmt)
    assert got == host_color_bytes(ids, offs, n_colors, fmt, f"fc_{fmt}")


def test_device_buffers_and_capacity():
    import torch
    res, ends = random_index_batch(9, 500)
    exp = S.format_index_results(res, ends, 31, 0)
    d_res = torch.from_numpy(res.view(np.int64)).cuda()
    d_ends = torch.from_numpy(ends.view(np.int64)).cuda()
    d_out = torch.zeros(len(exp), dtype=torch.uint8, device="cuda")
    nb = C.c_uint64()
    L = S.lib()
    st = torch.cuda.current_stream().cuda_stream
    rc = L.sbwt_format_index_results(d_res.data_ptr(), d_ends.data_ptr(), len(ends), 31, 0,
                                     d_out.data_ptr(), len(exp) - 1, C.byref(nb),
                                     S.DEVICE_POINTERS, 0, st)
    assert rc == S.E_CAPACITY and nb.value == len(exp)
    S.check(L.sbwt_format_index_results(d_res.data_ptr(), d_ends.data_ptr(), len(ends), 31, 0,
                                        d_out.data_ptr(), len(exp), C.byref(nb),
                                        S.DEVICE_POINTERS, 0, st))
    assert d_out.cpu().numpy().tobytes() == exp
    assert S.format_index_results(np.zeros(0, np.uint64), np.zeros(0, np.uint64), 31, 0) == b""


def _edge_values(rng, n, top):
    v = rng.integers(0, top, n, dtype=np.uint64)
    edges = [10 ** i + d for i in range(1, 20) for d in (-1, 0, 1)] + \
        [2 ** i + d for i in range(1, 40) for d in (-1, 0)]
    edges = np.array([e for e in edges if e < top], np.uint64)
    at = rng.random(n) < 0.5
    v[at] = rng.choice(edges, int(at.sum()))
    return v


@pytest.mark.parametrize("n_tokens", [0, 1, 2047, 2048, 2049, 4096, 9001])
@pytest.mark.parametrize("empty", [0, 3, 20_000])
@pytest.mark.parametrize("kind", ["index", "index_wide", "colors"])
def test_ascii_tiles_match_host_writer(n_tokens, empty, kind):
    """Token counts at the edges of tiles, reads that end on them, no or many
    empty reads before, between and after the others, digits of every length,
    and outputs and inputs at every alignment."""
    import torch
    rng = np.random.default_rng(n_tokens + empty)
    cuts = np.unique(np.concatenate([rng.integers(0, n_tokens + 1, 40), [0, n_tokens],
                                     np.arange(0, n_tokens, 2048)]))
    sizes = np.diff(cuts)
    where = np.concatenate([[0, len(sizes)], rng.integers(0, len(sizes) + 1, 2)])
    lines = list(sizes)
    for w in sorted(where)[::-1]:
        lines[w:w] = [0] * (empty // 4 + (empty > 0))
    lines = np.array(lines, np.int64)
    k = 5
    if kind == "colors":
        vals = _edge_values(rng, n_tokens, 1 << 32).astype(np.uint32)
        offs = np.concatenate([[0], np.cumsum(lines)]).astype(np.uint64)
        exp = host_color_bytes(vals, offs, 100, 0, "tiles_c")
    else:
        vals = _edge_values(rng, n_tokens, 1 << (32 if kind == "index" else 63))
        vals[rng.random(n_tokens) < 0.1] = O.NOT_FOUND
        vals[rng.random(n_tokens) < 0.1] = O.INVALID
        ends = np.cumsum(np.where(lines > 0, lines + k - 1, rng.integers(0, k, len(lines))))
        ends = ends.astype(np.uint64)
        exp = host_index_bytes(vals, ends, k, 0, "tiles_i")
    L, nb = S.lib(), C.c_uint64()
    for shift in range(0, 16, 5):
        lead = shift % 2  # tokens on and off a 16-byte boundary
        pad = np.concatenate([np.zeros(lead, vals.dtype), vals])
        d_v = torch.from_numpy(pad.view(np.int64 if vals.itemsize == 8 else np.int32)).cuda()
        out = torch.full((shift + len(exp) + 16,), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        if kind == "colors":  # offsets that do not start at 0
            d_o = torch.from_numpy((offs + np.uint64(lead)).view(np.int64)).cuda()
            torch.cuda.synchronize()
            rc = L.sbwt_format_color_results(d_v.data_ptr(), d_o.data_ptr(), len(lines), 100, 0,
                                             out.data_ptr() + shift, len(exp), C.byref(nb),
                                             S.DEVICE_POINTERS, 0, None)
        else:
            d_e = torch.from_numpy(ends.view(np.int64)).cuda()
            torch.cuda.synchronize()
            rc = L.sbwt_format_index_results(d_v.data_ptr() + 8 * lead, d_e.data_ptr(),
                                             len(lines), k, 0, out.data_ptr() + shift, len(exp),
                                             C.byref(nb), S.DEVICE_POINTERS, 0, None)
        assert rc == S.OK and nb.value == len(exp)
        h = out.cpu().numpy()
        assert h[shift:shift + len(exp)].tobytes() == exp
        assert (h[:shift] == 7).all() and (h[shift + len(exp):] == 7).all()


def _ascii_call(kind, vals, lines, cap, shift=0, k=5):
    """Lines of the given lengths through device pointers: (code, bytes needed,
    output with 16 bytes around it)."""
    import torch
    L, nb = S.lib(), C.c_uint64()
    d_v = torch.from_numpy(np.append(vals, vals.dtype.type(0)).view(
        np.int64 if vals.itemsize == 8 else np.int32)).cuda()
    out = torch.full((16 + shift + cap + 16,), 7, dtype=torch.uint8, device="cuda")
    if kind == "colors":
        d_o = torch.from_numpy(np.concatenate([[0], np.cumsum(lines)]).astype(np.int64)).cuda()
        torch.cuda.synchronize()
        rc = L.sbwt_format_color_results(d_v.data_ptr(), d_o.data_ptr(), len(lines), 100, 0,
                                         out.data_ptr() + 16 + shift, cap, C.byref(nb),
                                         S.DEVICE_POINTERS, 0, None)
    else:
        d_e = torch.from_numpy(np.cumsum(np.where(lines > 0, lines + k - 1, 1))).cuda()
        torch.cuda.synchronize()
        rc = L.sbwt_format_index_results(d_v.data_ptr(), d_e.data_ptr(), len(lines), k, 0,
                                         out.data_ptr() + 16 + shift, cap, C.byref(nb),
                                         S.DEVICE_POINTERS, 0, None)
    return rc, nb.value, out.cpu().numpy()


def _ascii_oracle(kind, vals, lines, name, k=5):
    if kind == "colors":
        offs = np.concatenate([[0], np.cumsum(lines)]).astype(np.uint64)
        return host_color_bytes(vals, offs, 100, 0, name)
    ends = np.cumsum(np.where(lines > 0, lines + k - 1, 1)).astype(np.uint64)
    return host_index_bytes(vals, ends, k, 0, name)


@pytest.mark.parametrize("kind", ["index", "index_wide", "colors"])
@pytest.mark.parametrize("n_tokens,empty,where", [
    (0, 8192, "first"), (0, 8193, "first"), (0, 300_000, "first"), (1, 300_000, "first"),
    (1, 300_000, "last"), (2048, 40_000, "first"), (2048, 40_000, "last"),
    (6000, 200_000, "between"), (6000, 60_000, "spread"), (70_000, 1_000_000, "spread"),
    (5000, 0, "none")])
def test_ascii_of_mostly_empty_reads(n_tokens, empty, where, kind):
    """Batches of which few reads have a token: tiles with more lines than shared
    memory holds, whose empty reads lie before, after and between the tokens, in
    one stretch or many; exact and large capacities, and one byte too few."""
    rng = np.random.default_rng(n_tokens + empty)
    n_lines = min(n_tokens, max(1, n_tokens // 3))
    cuts = np.sort(rng.choice(np.arange(1, max(n_tokens, 2)), max(n_lines - 1, 0), replace=False))
    sizes = np.diff(np.concatenate([[0], cuts, [n_tokens]])) if n_tokens else np.zeros(0, np.int64)
    at = {"first": 0, "last": len(sizes), "between": len(sizes) // 2}.get(where, 0)
    lines = np.insert(sizes, at, np.zeros(empty, np.int64))
    if where == "spread":
        lines = np.zeros(len(sizes) + empty, np.int64)
        lines[np.sort(rng.choice(len(lines), len(sizes), replace=False))] = sizes
    top = {"index": 1 << 32, "index_wide": 1 << 63, "colors": 1 << 32}[kind]
    vals = _edge_values(rng, n_tokens, top)
    if kind == "index_wide":  # 16 digits and more: tiles are big without empty reads too
        vals = np.maximum(vals, np.uint64(10 ** 16))
    if kind == "colors":
        vals = vals.astype(np.uint32)
    else:
        vals[rng.random(n_tokens) < 0.1] = O.NOT_FOUND
    exp = _ascii_oracle(kind, vals, lines, "mostly_empty")
    for cap, shift in ((len(exp), 0), (len(exp), 5), (len(exp) + (40 << 20), 11)):
        rc, need, out = _ascii_call(kind, vals, lines, cap, shift)
        assert rc == S.OK and need == len(exp)
        lo = 16 + shift
        assert out[lo:lo + need].tobytes() == exp
        assert (out[:lo] == 7).all() and (out[lo + need:] == 7).all()
    rc, need, out = _ascii_call(kind, vals, lines, len(exp) - 1)
    assert rc == S.E_CAPACITY and need == len(exp) and (out == 7).all()


@pytest.mark.parametrize("kind", ["index", "colors"])
@pytest.mark.parametrize("empty", [0, 300_000])
@pytest.mark.parametrize("top", [1 << 8, 1 << 32])
def test_ascii_of_a_large_batch(top, empty, kind):
    """More tiles than are written before the host knows their count, by a
    capacity that bounds the count (short tokens) and by one from which on it is
    read back."""
    rng = np.random.default_rng(empty + 1)
    sizes = rng.integers(1, 200, 26_000)
    lines = np.insert(sizes, rng.integers(0, len(sizes), empty), 0)
    vals = _edge_values(rng, int(sizes.sum()), top)
    if kind == "colors":
        vals = vals.astype(np.uint32)
    exp = _ascii_oracle(kind, vals, lines, "large")
    assert len(vals) > 1100 * 2048 and (len(exp) > 16 << 20) == (top > 1 << 8)
    rc, need, out = _ascii_call(kind, vals, lines, len(exp), 3)
    assert rc == S.OK and need == len(exp)
    assert out[19:19 + need].tobytes() == exp
    assert (out[:19] == 7).all() and (out[19 + need:] == 7).all()
