"""Read search between host buffers: chars staged, results mapped and widened by
slices of a chunk on host threads."""
import numpy as np
import pytest

import sbwt_b200 as S
import sbwt_tools as T
from helpers import TMP

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    import torch
    g = T.gen_genomes(11, 4, 200_000, 2, 0.02, 0.0, 0.0)
    path = TMP / "host_slices.sbwt"
    T.build_sbwt(g, 31, str(path))
    idx = S.SbwtIndex.open(path)
    chars, ends = T.gen_reads(3, g, 60_000, 0.9, 120, 0.4, 20, 600, 0.01, 0.001)
    out = torch.empty(len(chars), dtype=torch.int64, device="cuda")
    n = idx.search_reads(torch.from_numpy(chars.copy()).cuda(),
                         torch.from_numpy(ends.view(np.int64).copy()).cuda(), out=out)
    exp = out[:n].cpu().numpy().view(np.uint64)
    assert n > 4 << 20  # slices of 2^20 k-mers: several
    yield idx, chars, ends, exp
    idx.close()


# the whole batch, and chunks of one, two and three slices; results at and off a
# page and its neighbours
@pytest.mark.parametrize("chunk", [0, 900_000, 2_900_000, 4_000_001])
@pytest.mark.parametrize("offset", [0, 1, 511, 262_143])
def test_slices_of_a_chunk(case, chunk, offset):
    idx, chars, ends, exp = case
    room = np.full(len(exp) + offset + 7, 77, np.uint64)
    out = room[offset:offset + len(exp)]
    try:
        S.set_launch_config(chunk_chars=chunk)
        got = idx.search_reads(chars, ends, out=out)
    finally:
        S.set_launch_config()
    assert np.array_equal(got, exp)
    assert (room[:offset] == 77).all() and (room[offset + len(exp):] == 77).all()


def test_slices_then_an_error(case):
    """A buffer too small and unordered ends are reported, with the chunks
    before them on their threads, and the next call is whole again."""
    idx, chars, ends, exp = case
    S.set_launch_config(chunk_chars=3_000_000)
    try:
        room = np.full(len(exp), 77, np.uint64)
        with pytest.raises(S.SbwtError):
            idx.search_reads(chars, ends, out=room[:-1])
        assert room[-1] == 77
        bad = ends.copy()
        bad[-2] = bad[-1] + np.uint64(5)
        with pytest.raises(S.SbwtError):
            idx.search_reads(chars, bad, out=room)
        assert np.array_equal(idx.search_reads(chars, ends), exp)
    finally:
        S.set_launch_config()
