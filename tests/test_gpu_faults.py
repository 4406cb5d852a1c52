"""Calls whose device work fails report it themselves and leave the cell in
a state that the next calls answer from correctly.  The failures are made on
the host (dct_b200_fault_inject); nothing fails on the device."""
import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
from oracle.dp_oracle import OracleBackend

pytestmark = pytest.mark.gpu

STREAMED, BARRIER, PINNED = 0, 1, 2      # dct_b200_fault_inject kinds


@pytest.fixture
def streamed_cell(monkeypatch):
    """A ternary cell whose plans stream, untuned, at a 60% cover."""
    monkeypatch.setenv("CC_TMA", "1")
    monkeypatch.setenv("CC_TUNE", "0")
    monkeypatch.setenv("DCT_SET_GATHER", "0")
    axes, R = [3] * 12, 4
    size = 3 ** 12
    code = np.random.default_rng(4).choice(size, 60, replace=False)
    with GpuBackend(axes, R) as b:
        yield b, code, OracleBackend(axes, R)
        b._lib.dct_b200_fault_inject(STREAMED, 0)


def test_a_streamed_time_out_is_the_failing_transforms_error(streamed_cell):
    b, code, o = streamed_cell
    b.recount(code)
    o.recount(code)
    b._lib.dct_b200_fault_inject(STREAMED, 1)
    with pytest.raises(RuntimeError):
        b.gain_map()
    b.gain_map()                         # reported once, by that call
    o.gain_map()
    assert np.array_equal(b.map_all(), o.map)


def test_a_streamed_time_out_is_the_failing_gathers_error(streamed_cell,
                                                          monkeypatch):
    """Untuned (straight after a recount) and with the plan of an earlier
    gain map: the call answered by one transform reports, the next one and
    the next transform are right."""
    b, code, o = streamed_cell
    monkeypatch.setenv("CC_GATHER_TRANSFORM", "1")
    b.recount(code)
    o.recount(code)
    cands = np.random.default_rng(1).integers(0, 3 ** 12, 5000)
    want = o.ball_gather(cands[:200], 0)
    for _ in range(2):
        b._lib.dct_b200_fault_inject(STREAMED, 1)
        with pytest.raises(RuntimeError):
            b.ball_gather(cands, 0)
        assert np.array_equal(b.ball_gather(cands, 0)[:200], want)
        b.gain_map()
    o.gain_map()
    assert np.array_equal(b.map_all(), o.map)


def test_a_streamed_time_out_is_the_failing_batch_calls_error(monkeypatch):
    """A step of one launch per pass and a greedy whose gain rebuilds stream:
    each reports, and the next step and greedy are the oracle's."""
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    monkeypatch.setenv("CC_TUNE", "0")
    monkeypatch.setenv("CC_GREEDY_REBUILD", "1")
    axes, R = (3,) * 11, 3
    code = np.random.default_rng(6).choice(3 ** 11, 80, replace=False)
    o = OracleBackend(list(axes), R)
    o.recount(code)
    with BatchEngine() as e:
        e.add("hamming", axes, R, code)
        e.build(48)
        e.set_table(0, wide_table(axes, R, "hamming"))
        lib = e._lib
        for mode in (0, 1):
            lib.dct_b200_fault_inject(STREAMED, 1)
            assert e.run_rc(1) == -8
            e.run(mode)
            assert np.array_equal(e.cnt(0), o.read_cnt())
            lib.dct_b200_fault_inject(STREAMED, 1)
            with pytest.raises(RuntimeError):
                e.greedy([0], [4])
        lib.dct_b200_fault_inject(STREAMED, 0)
        e.run(0)
        assert e.scalars()[0, 0] == o.uncovered()
        (placed, deficit), = e.greedy([0], [4])
        o.ball_update(placed, 1)
        assert deficit == o.uncovered()
        assert np.array_equal(e.cnt(0), o.read_cnt())


def refuses(b, w):
    """Every call that reads cnt is refused."""
    calls = [lambda: b.gain_map(), lambda: b.loss_map(), lambda: b.uncovered(),
             lambda: b.ball_gather(w, 0), lambda: b.ball_update(w, 1),
             lambda: b.ball_update_delta(w, 1), lambda: b.read_cnt(),
             lambda: b.swap_eval(w, w), lambda: b.greedy_fill_device(1)]
    for i, call in enumerate(calls):
        with pytest.raises(RuntimeError):
            call()
            raise AssertionError(f"call {i} answered")


@pytest.mark.parametrize("axes,R", [([2] * 14, 2), ([3] * 9, 2)])
def test_a_greedy_that_times_out_stops_and_asks_for_a_recount(axes, R,
                                                              monkeypatch):
    """A barrier time-out ends the greedy at that launch: the launch after it
    would start on a half-done step.  cnt then lies between two states: no
    call answers from it, nor from a list of the deficient words made before
    the greedy, until a recount."""
    monkeypatch.setenv("CC_GREEDY_REBUILD", "0")
    monkeypatch.setenv("DCT_SET_GATHER", "2")
    size = int(np.prod(axes))
    code = np.random.default_rng(2).choice(size, 20, replace=False)
    o = OracleBackend(axes, R)
    o.recount(code)
    cands = np.arange(0, size, 7)
    with GpuBackend(axes, R) as b:
        b.recount(code)
        before = b.uncovered()
        assert np.array_equal(b.ball_gather(cands, 0), o.ball_gather(cands, 0))
        b._lib.dct_b200_fault_inject(BARRIER, 1)
        with pytest.raises(RuntimeError):
            b.greedy_fill_device(60)
        refuses(b, code[:3])
        b.recount(code)
        assert b.uncovered() == before == o.uncovered()
        placed, deficit = b.greedy_fill_device(60)
        o.ball_update(placed, 1)
        assert deficit == o.uncovered() == b.uncovered()
        b.ball_update(placed, -1)        # they are active words
        assert b.uncovered() == before


def test_a_recount_that_times_out_asks_for_a_recount(streamed_cell):
    b, code, o = streamed_cell
    b.recount(code)
    b._lib.dct_b200_fault_inject(STREAMED, 1)
    with pytest.raises(RuntimeError):
        b.recount(code[:40])
    refuses(b, code[:2])
    b.recount(code[:40])
    o.recount(code[:40])
    assert np.array_equal(b.read_cnt(), o.read_cnt())
    b.ball_update(code[:2], -1)
    o.ball_update(code[:2], -1)
    assert b.uncovered() == o.uncovered()


def test_a_greedy_rebuild_that_times_out_is_the_greedys_error(streamed_cell,
                                                              monkeypatch):
    b, code, o = streamed_cell
    monkeypatch.setenv("CC_GREEDY_REBUILD", "1")
    b.recount(code)
    b.gain_map()
    b._lib.dct_b200_fault_inject(STREAMED, 2)
    with pytest.raises(RuntimeError):
        b.greedy_fill_device(3)
    refuses(b, code[:2])
    b.recount(code)
    o.recount(code)
    placed, deficit = b.greedy_fill_device(3)
    o.ball_update(placed, 1)
    assert deficit == o.uncovered()


@pytest.mark.parametrize("rebuild", ["0", "1"])
def test_an_error_of_an_earlier_step_is_not_a_greedys(rebuild, monkeypatch):
    """The dependency-wait self-test leaves its error word; the step of one
    launch per pass after it is right, and so is the greedy from that step."""
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    monkeypatch.setenv("CC_GREEDY_REBUILD", rebuild)
    axes, R = (2,) * 13, 1
    code = np.random.default_rng(7).choice(2 ** 13, 30, replace=False)
    o = OracleBackend(list(axes), R)
    o.recount(code)
    with BatchEngine() as e:
        e.add("hamming", axes, R, code)
        e.build(16)
        e.set_table(0, wide_table(axes, R, "hamming"))
        assert e.run_rc(2) == -7
        e.run(1)
        (placed, deficit), = e.greedy([0], [5])
        assert len(placed) == 5
        o.ball_update(placed, 1)
        assert deficit == o.uncovered()
        assert np.array_equal(e.cnt(0), o.read_cnt())


def test_a_code_that_is_refused_room_leaves_the_staged_one():
    """A second, larger code whose pinned room is refused: the recount is of
    the code staged before it, whose words can then be taken out."""
    axes, R = [3] * 9, 2
    rng = np.random.default_rng(3)
    first, large = (rng.choice(3 ** 9, m, replace=False) for m in (30, 9000))
    o = OracleBackend(axes, R)
    with GpuBackend(axes, R) as b:
        b.recount(rng.choice(3 ** 9, 50, replace=False))
        b.stage_code(first)
        b._lib.dct_b200_fault_inject(PINNED, 1)
        with pytest.raises(RuntimeError):
            b.stage_code(large)
        assert b._lib.dct_transform(0, 2) == 0
        o.recount(first)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        b.ball_update(first[:5], -1)
        o.ball_update(first[:5], -1)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        with pytest.raises(RuntimeError):
            b.ball_update(first[:1], -1)
        b.recount(large)                 # with room it is staged
        o.recount(large)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
