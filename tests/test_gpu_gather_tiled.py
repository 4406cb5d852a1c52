"""The tiled gather (a block walks a tile of the support table for a group
of candidates), with and without the predicate bit plane, against the
oracle and against the per-word walk, for Hamming, Lee, torus and
mixed-radix cells, mu = 1 and 2, every role."""
import ctypes

import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
from coldcore_b200.patterns import wide_table
from oracle.dp_oracle import OracleBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problem,axes,R,mu", [
    ("hamming", [3] * 8, 3, 1), ("hamming", [3] * 12, 4, 1),
    ("hamming", [2, 3, 4, 5, 6, 7], 3, 2), ("lee", [7] * 6, 3, 1),
    ("torus_linf", [5, 6, 7], 1, 1), ("hamming", [2] * 16, 5, 2)])
def test_tiled_gather_matches(monkeypatch, problem, axes, R, mu):
    size = int(np.prod(axes))
    rng = np.random.default_rng(len(axes) * 7 + R)
    code = rng.choice(size, size=max(3, size // 40), replace=False)
    o = OracleBackend(axes, R, problem=problem, mu=mu)
    o.recount(code)
    cands = rng.integers(0, size, 333).astype(np.int64)
    with GpuBackend(axes, R, problem=problem, mu=mu) as b:
        b.recount(code)
        for role in (0, 1, 2):
            want = o.ball_gather(cands, role)
            monkeypatch.setenv("CC_GATHER_TILED", "1")
            monkeypatch.setenv("CC_GATHER_BITS", "1")
            bits = b.ball_gather(cands, role)
            monkeypatch.setenv("CC_GATHER_BITS", "0")
            tiled = b.ball_gather(cands, role)
            monkeypatch.setenv("CC_GATHER_TILED", "0")
            walk = b.ball_gather(cands, role)
            assert np.array_equal(bits, want), role
            assert np.array_equal(tiled, want), role
            assert np.array_equal(walk, want), role


@pytest.mark.parametrize("problem,axes,R,mu", [
    ("hamming", [3] * 12, 4, 1), ("hamming", [3] * 9, 3, 2),
    ("hamming", [2] * 16, 3, 1), ("hamming", [2] * 15, 5, 2),
    ("hamming", [2, 3, 4, 5, 6, 7], 3, 2), ("lee", [7] * 6, 4, 1),
    ("hamming", [5] * 7, 3, 1), ("hamming", [3] * 8, 2, 1)])
def test_gather_by_transform_matches(monkeypatch, problem, axes, R, mu):
    """A call answered by one transform of the predicate: every role and a
    literal count, more candidates than a staging chunk, the map of an
    earlier transform left as it was, and exact layers left alone."""
    size = int(np.prod(axes))
    rng = np.random.default_rng(len(axes) * 5 + R)
    code = rng.choice(size, size=max(3, size // 60), replace=False)
    o = OracleBackend(axes, R, problem=problem, mu=mu)
    o.recount(code)
    cands = rng.integers(0, size, 70001).astype(np.int64)
    some = cands[-300:]
    monkeypatch.setenv("CC_GATHER_TRANSFORM", "1")
    with GpuBackend(axes, R, problem=problem, mu=mu) as b:
        b.recount(code)
        b.gain_map()
        before = b.map_all()
        for role in (0, 1, 2):
            got = b.ball_gather(cands, role)
            assert np.array_equal(got[-300:], o.ball_gather(some, role)), role
            monkeypatch.setenv("CC_GATHER_TRANSFORM", "0")
            assert np.array_equal(got, b.ball_gather(cands, role)), role
            monkeypatch.setenv("CC_GATHER_TRANSFORM", "1")
        assert np.array_equal(b.map_all(), before)
        b.stage_code(code)
        b.layers_map(0)
        at = b.layers_at(some)
        b.ball_gather(cands, 0)
        assert np.array_equal(b.layers_at(some), at)


def second_table(b, tbl):
    """dct_set_tbl2 from the rows of a wide table."""
    mask = np.zeros(len(tbl), dtype=np.uint16)
    offs = np.zeros(len(tbl), dtype=np.uint64)
    for k in range(tbl.shape[1]):
        pos, dl = tbl[:, k] >> 24, tbl[:, k] & 0xFFFFFF
        used = dl > 0
        mask[used] |= (1 << pos[used]).astype(np.uint16)
        offs[used] |= dl[used].astype(np.uint64) << (
            4 * pos[used]).astype(np.uint64)
    p = ctypes.POINTER
    assert b._lib.dct_set_tbl2(
        mask.ctypes.data_as(p(ctypes.c_uint16)),
        offs.ctypes.data_as(p(ctypes.c_uint64)), len(tbl)) == 0


def test_second_table_of_other_patterns(monkeypatch):
    """dct_use_fmt(1) with a table that is not the ball: large gathers answer
    from that table as small ones do, and a greedy never places a word that
    is active although the table did not cover it."""
    monkeypatch.setenv("DCT_SET_GATHER", "0")
    monkeypatch.setenv("CC_GATHER_TRANSFORM", "1")
    axes, R = [3] * 9, 3
    size = 3 ** 9
    tbl = wide_table(axes, R, "hamming")
    other = tbl.copy()
    other[::3] = tbl[2]                  # pattern 0, the centre, too
    rng = np.random.default_rng(9)
    cands = rng.integers(0, size, 30000)
    with GpuBackend(axes, R) as b:
        second_table(b, other)
        b.recount(rng.choice(size, 40, replace=False))
        assert b._lib.dct_use_fmt(1) == 0
        small = np.concatenate([b.ball_gather(cands[i:i + 6000], 0)
                                for i in range(0, len(cands), 6000)])
        assert np.array_equal(b.ball_gather(cands, 0), small)
        assert b._lib.dct_use_fmt(0) == 0
        assert not np.array_equal(b.ball_gather(cands, 0), small)
    # word 0 is active, yet all but one word of its ball is uncovered
    monkeypatch.setenv("DCT_SET_GATHER", "1")
    axes, R = [3] * 6, 1
    tbl = wide_table(axes, R, "hamming")
    tbl[:] = tbl[2]
    x = np.arange(3 ** 6)
    weight = sum((x // 3 ** j % 3 != 0).astype(int) for j in range(6))
    with GpuBackend(axes, R) as b:
        second_table(b, tbl)
        b.recount(x[weight >= 3])
        assert b._lib.dct_use_fmt(1) == 0
        b.ball_update([0], +1)
        assert b._lib.dct_use_fmt(0) == 0
        assert b.uncovered() == 12 == b.ball_gather([0], 0)[0]
        placed, _ = b.greedy_fill_device(12)
        assert len(placed) and 0 not in placed


@pytest.mark.parametrize("problem,axes,R,mu,tuned,transform", [
    ("hamming", [3] * 12, 4, 1, False, True),      # padded, streamed
    ("hamming", [3] * 13, 4, 2, False, True),
    ("hamming", [4] * 9, 4, 1, False, True),
    ("hamming", [5] * 8, 4, 2, False, True),
    ("lee", [7] * 6, 4, 1, False, True),
    ("hamming", [2] * 16, 3, 1, False, True),      # streamed, unpadded
    ("hamming", [2] * 18, 3, 1, False, False),     # more than 16 axes
    ("hamming", [3] * 14, 4, 1, True, True),       # tuned, its map redirected
    ("hamming", [4] * 11, 3, 2, True, None),       # whichever plan won
    ("hamming", [3] * 11, 3, 1, False, False),     # pitched planes too wide
    ("hamming", [3] * 12, 2, 1, False, False),     # three layers: no room
])
def test_which_large_gathers_one_transform_answers(monkeypatch, problem, axes,
                                                   R, mu, tuned, transform):
    """The route of a large gather (gpu_stats) and its counts: straight after
    a recount, on the plan made for it, or on the tuned plan of an earlier
    gain map, which stays as it was."""
    from oracle.cport import CPortCell
    monkeypatch.setenv("CC_GATHER_TRANSFORM", "1")
    monkeypatch.setenv("DCT_SET_GATHER", "0")
    size = int(np.prod(axes))
    rng = np.random.default_rng(len(axes) + R)
    code = rng.choice(size, size // 700, replace=False)
    o = CPortCell(axes, R, problem, mu=mu)
    o.recount(code)
    o.gain_map()
    gain = o.map.copy()
    o.loss_map()
    cands = rng.integers(0, size, 70001)
    with GpuBackend(axes, R, problem=problem, mu=mu) as b:
        b.recount(code)
        if tuned:
            b.gain_map()
        for role, want in ((0, gain), (1, o.map)):
            before = b.gpu_stats()["gather_transform"]
            assert np.array_equal(b.ball_gather(cands, role), want[cands])
            if transform is not None:
                used = b.gpu_stats()["gather_transform"] - before
                assert used == (1 if transform else 0)
        if tuned:
            assert np.array_equal(b.map_all(), gain)
        assert np.array_equal(b.read_cnt(), o.cnt)
