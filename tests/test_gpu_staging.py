"""The staged code, the active multiset and the map queries' results on the
host: what a recount stages, which updates the multiset then accepts, and
the answers that pass the staging buffers' first copy."""
import ctypes
from collections import Counter

import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
from oracle.dp_oracle import OracleBackend

pytestmark = pytest.mark.gpu


def test_a_code_staged_after_a_recount_waits_for_its_own():
    """Updates go to the recounted multiset, whatever has been staged since;
    the staged code becomes the multiset with its recount."""
    axes, R, size = [3] * 8, 2, 3 ** 8
    rng = np.random.default_rng(1)
    first = rng.choice(size, 40, replace=False)
    second = np.setdiff1d(rng.choice(size, 70, replace=False), first)
    o = OracleBackend(axes, R)
    o.recount(first)
    with GpuBackend(axes, R) as b:
        b.recount(first)
        for code in (second[:20], second):           # staged twice
            b.stage_code(code)
        with pytest.raises(RuntimeError):
            b.ball_update(second[:1], -1)
        b.ball_update(first[:7], -1)
        o.ball_update(first[:7], -1)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        with pytest.raises(RuntimeError):
            b.ball_update(first[:1], -1)
        assert b._lib.dct_transform(0, 2) == 0
        o.recount(second)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        b.ball_update(second, -1)
        assert not b.read_cnt().any()


def test_updates_that_cancel_and_repeats():
    """A thousand updates against a plain multiset: words put in and taken
    out again, repeats, a word of the code taken out and put back; what the
    multiset does not hold is refused and changes nothing."""
    axes, R, size = [4] * 5, 1, 4 ** 5
    rng = np.random.default_rng(2)
    code = rng.integers(0, size, 60)                 # repeats among them
    held = Counter(code.tolist())
    o = OracleBackend(axes, R)
    o.recount(code)
    with GpuBackend(axes, R) as b:
        b.recount(code)
        pool = np.concatenate([code, rng.integers(0, size, 40)])
        for step in range(1000):
            words = rng.choice(pool, rng.integers(1, 5))
            delta = int(rng.choice([-1, 1]))
            want = Counter(words.tolist())
            if delta < 0 and any(held[w] < k for w, k in want.items()):
                with pytest.raises(RuntimeError):
                    b.ball_update(words, -1)
                continue
            b.ball_update(words, delta)
            o.ball_update(words, delta)
            for w, k in want.items():
                held[w] += delta * k
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        rest = np.array(sorted(held.elements()), dtype=np.int64)
        b.ball_update(rest, -1)                      # exactly these are held
        assert not b.read_cnt().any()


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("cap", [1, 32767, 32768, 32769, 60000, 200000])
def test_extractions_around_the_first_copy(cap, wide):
    """Fewer, as many and more entries than come back with their count."""
    axes, R, size = [3] * 11, 2, 3 ** 11
    code = np.random.default_rng(3).choice(size, 300, replace=False)
    o = OracleBackend(axes, R)
    o.recount(code)
    o.gain_map()
    order = np.sort(o.map)[::-1]
    with GpuBackend(axes, R, extract_cap=1 << 18) as b:
        b.recount(code)
        b.gain_map()
        for thr in sorted({1, int(order[32768]), int(order[32767]),
                           int(order[0]), int(order[0]) + 1}):
            if wide:
                idx = np.full(cap, -1, dtype=np.int64)
                val = np.full(cap, -1, dtype=np.int32)
                found = b._lib.dct_map_extract64(
                    thr, idx.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                    val.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), cap)
                m = min(found, cap)
                assert (idx[m:] == -1).all() and (val[m:] == -1).all()
                idx, val = idx[:m], val[:m]
            else:
                idx, val, found = b.map_extract(thr, cap=cap)
            assert found == np.count_nonzero(o.map >= thr)
            assert len(idx) == min(found, cap) == len(np.unique(idx))
            assert np.array_equal(val, o.map[idx]) and (val >= thr).all()


@pytest.mark.parametrize("nbins", [1, 3, 1000, 1024, 4095, 4096])
def test_histogram_bins_at_the_edges_of_the_division(nbins):
    """Counter values up to 65,535 binned by (v - 1) * nbins // vmax: vmax a
    power of two and one to either side, beside the largest whose product
    with nbins is below 2^31, and above it."""
    size = 2 ** 12
    mult = np.unique(np.concatenate(
        [2 ** np.arange(12), 2 ** np.arange(1, 12) - 1,
         2 ** np.arange(1, 12) + 1, [2900, 3583]]))
    words = np.arange(len(mult)) * 64
    with GpuBackend([2] * 12, 1) as b:
        # balls of radius 1 around words 64 apart: sums of the multiplicities
        b.stage_code(np.repeat(words, mult))
        assert b._lib.dct_transform(0, 1) == 0
        values = b.map_all().astype(np.int64)
        assert values.max() > 4096 and len(values) == size
        top = (2 ** 31 - 1) // nbins
        for vmax in {1, 2, 3, int(values.max()) - 1, int(values.max()),
                     int(values.max()) + 1, min(top, 2 ** 31 - 2) - 1,
                     min(top, 2 ** 31 - 2), min(top, 2 ** 31 - 2) + 1,
                     2 ** 31 - 1, *(2 ** k + d for k in range(2, 31)
                                    for d in (-1, 0, 1))}:
            pos = values[values > 0]
            want = np.bincount(np.minimum((pos - 1) * nbins // vmax,
                                          nbins - 1), minlength=nbins)
            assert np.array_equal(b.map_hist(nbins, vmax), want), vmax
