"""Color counters at the edges of their bit planes, rounds and tiles: device
and host calls equal to the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import sbwt_b200 as S
import sbwt_tools as T
from helpers import TMP

pytestmark = pytest.mark.gpu

# k-mers per read: rounds of 128, trees of 8 rows, 8 planes (255 / 256)
SPANS = [0, 1, 7, 8, 9, 31, 32, 33, 127, 128, 129, 254, 255, 256, 257, 700]


@pytest.mark.parametrize("n_colors", [1, 2, 63, 64, 65, 2047, 2048, 2049])
@pytest.mark.parametrize("long_read", [False, True])  # 16 planes hold 65,535
def test_counters_match_oracle(n_colors, long_read):
    import torch
    g = T.gen_genomes(31, n_colors, 150, min(n_colors, 5), 0.01, 0.04, 0.0)
    sp, cp = TMP / f"cc_{n_colors}.sbwt", TMP / f"cc_{n_colors}.tcolors"
    T.build_colored(g, 31, str(sp), str(cp))
    idx, ci = S.SbwtIndex.open(sp), S.ColorIndex.open(cp)
    nodes = idx.search_reads(g.chars, np.cumsum(g.lens).astype(np.uint64))
    rng = np.random.default_rng(n_colors)
    spans = SPANS + ([65_535, 65_536] if long_read else [])
    found = []
    for i, n in enumerate(spans):  # neighbours, repeats of one k-mer, or any k-mers
        if i % 3 == 0:
            found.append(np.resize(nodes[int(rng.integers(0, len(nodes))):], n))
        elif i % 3 == 1:
            found.append(np.repeat(rng.choice(nodes, (n + 39) // 40), 40)[:n])
        else:
            found.append(rng.choice(nodes, n))
    flat = np.concatenate(found).astype(np.uint64)
    offs = np.concatenate([[0], np.cumsum(spans)]).astype(np.uint64)
    oc = O.OracleColors(O.ColorsFile.read(cp))
    zero = np.zeros(len(spans), np.uint64)
    rows, exp = oc.pseudoalign(found, zero, zero, 0.6, want_counts=True)
    assert np.array_equal(ci.counts(flat, offs).astype(np.uint64), exp)
    assert ci.pseudoalign(flat, offs, tau=0.6)[0] == rows
    d_flat, d_offs = (torch.from_numpy(x.view(np.int64).copy()).cuda() for x in (flat, offs))
    for pad in (0, 1):  # counts on and off a 16-byte boundary
        buf = torch.full((len(spans) * n_colors + pad + 1,), -7, dtype=torch.int32, device="cuda")
        S.check(S.lib().sbwt_color_counts(ci._h, d_flat.data_ptr(), d_offs.data_ptr(), len(spans),
                                          buf.data_ptr() + 4 * pad, S.DEVICE_POINTERS, None))
        got = buf.cpu().numpy()
        assert np.array_equal(got[pad:-1].astype(np.uint64).reshape(exp.shape), exp)
        assert got[-1] == -7 and (pad == 0 or got[0] == -7)
    n_ids = sum(map(len, rows))
    io = torch.zeros(len(spans) + 1, dtype=torch.int64, device="cuda")
    for cap in (n_ids, n_ids - 1):
        ids = torch.full((n_ids + 1,), -7, dtype=torch.int32, device="cuda")
        rc = S.lib().sbwt_pseudoalign(ci._h, d_flat.data_ptr(), d_offs.data_ptr(), None, None,
                                      len(spans), C.c_double(0.6), S.DEVICE_POINTERS,
                                      ids.data_ptr(), max(cap, 0), io.data_ptr(), None)
        assert rc == (S.OK if cap == n_ids else S.E_CAPACITY)
        assert np.array_equal(np.diff(io.cpu().numpy()), [len(r) for r in rows])
        if rc == S.OK:
            h = ids.cpu().numpy()
            assert h[:n_ids].tolist() == sum(rows, []) and h[n_ids] == -7


def test_decreasing_device_offsets_are_an_error():
    import torch
    g = T.gen_genomes(31, 2, 150, 2, 0.01, 0.04, 0.0)
    sp, cp = TMP / "cc_bad.sbwt", TMP / "cc_bad.tcolors"
    T.build_colored(g, 31, str(sp), str(cp))
    ci = S.ColorIndex.open(cp)
    vals = torch.zeros(8, dtype=torch.int64, device="cuda")
    out = torch.zeros(64, dtype=torch.int32, device="cuda")
    for offs in ([0, 8, 4, 8], [0, 1000, 4, 8], [8, 4, 4, 8]):
        d = torch.tensor(offs, dtype=torch.int64, device="cuda")
        rc = S.lib().sbwt_color_counts(ci._h, vals.data_ptr(), d.data_ptr(), 3, out.data_ptr(),
                                       S.DEVICE_POINTERS, None)
        assert rc == S.E_INVALID


@pytest.mark.parametrize("n_colors", [40, 2100])
@pytest.mark.parametrize("share", [0.001, 0.3, 1.0])
def test_long_reads_among_short_ones(n_colors, share):
    """Device batches whose longer reads take a second launch: none but one, some
    and all of them long, in any order; a value past the index in a read of
    either kind is an error, and the next call is right."""
    import torch
    g = T.gen_genomes(37, n_colors, 150, 5, 0.01, 0.04, 0.0)
    sp, cp = TMP / f"cl_{n_colors}.sbwt", TMP / f"cl_{n_colors}.tcolors"
    T.build_colored(g, 31, str(sp), str(cp))
    idx, ci = S.SbwtIndex.open(sp), S.ColorIndex.open(cp)
    nodes = idx.search_reads(g.chars, np.cumsum(g.lens).astype(np.uint64))
    rng = np.random.default_rng(n_colors)
    spans = rng.integers(0, 130, 2000)
    at = rng.choice(2000, max(1, int(2000 * share)), replace=False)
    spans[at] = rng.integers(256, 400, len(at))
    is_short = np.flatnonzero((spans > 0) & (spans < 256))
    bad_reads = [int(at[0])] + [int(r) for r in is_short[:1]]
    flat = np.concatenate([np.resize(nodes[int(rng.integers(0, len(nodes))):], n) for n in spans])
    offs = np.concatenate([[0], np.cumsum(spans)]).astype(np.uint64)
    oc = O.OracleColors(O.ColorsFile.read(cp))
    zero = np.zeros(len(spans), np.uint64)
    rows, exp = oc.pseudoalign([flat[offs[r]:offs[r + 1]] for r in range(2000)], zero, zero, 0.6,
                               want_counts=True)
    n_ids = sum(map(len, rows))
    d_offs = torch.from_numpy(offs.view(np.int64).copy()).cuda()
    for bad in (None, *bad_reads, None):
        vals = flat.copy()
        if bad is not None:
            vals[offs[bad]] = 1 << 40
        d_vals = torch.from_numpy(vals.view(np.int64).copy()).cuda()
        io = torch.zeros(len(spans) + 1, dtype=torch.int64, device="cuda")
        ids = torch.full((n_ids + 1,), -7, dtype=torch.int32, device="cuda")
        counts = torch.full((2000 * n_colors + 1,), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = S.lib().sbwt_pseudoalign(ci._h, d_vals.data_ptr(), d_offs.data_ptr(), None, None, 2000,
                                      C.c_double(0.6), S.DEVICE_POINTERS, ids.data_ptr(), n_ids,
                                      io.data_ptr(), None)
        rc2 = S.lib().sbwt_color_counts(ci._h, d_vals.data_ptr(), d_offs.data_ptr(), 2000,
                                        counts.data_ptr(), S.DEVICE_POINTERS, None)
        if bad is not None:
            assert rc == S.E_INVALID and rc2 == S.E_INVALID
            continue
        assert rc == S.OK and rc2 == S.OK
        h = ids.cpu().numpy()
        assert h[:n_ids].tolist() == sum(rows, []) and h[n_ids] == -7
        assert np.array_equal(np.diff(io.cpu().numpy()), [len(r) for r in rows])
        h = counts.cpu().numpy()
        assert np.array_equal(h[:-1].astype(np.uint64).reshape(exp.shape), exp) and h[-1] == -7
