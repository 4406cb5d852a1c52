"""Device-side exact greedy repair (``dct_b200_greedy_fill``) on the B200
against the brute-force exact greedy of the oracle: the same words in the
same order (largest exact gain, ties to the smallest index), the same
deficit, the same counters afterwards."""
import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
from oracle.dp_oracle import OracleBackend, exact_greedy

pytestmark = pytest.mark.gpu

CELLS = [("hamming", [3] * 7, 2, 1), ("hamming", [4, 3, 5, 2, 3], 2, 2),
         ("hamming", [2] * 11, 3, 1), ("lee", [5, 6, 7, 4], 2, 1),
         ("lee", [4] * 5, 3, 2), ("torus_linf", [7, 9, 11], 2, 1),
         ("torus_linf", [5, 5, 5], 1, 2), ("grid_linf", [4, 5, 6], 2, 1),
         ("grid_linf", [3, 3, 8], 1, 1), ("grid_linf", [6, 7], 3, 1)]


@pytest.mark.parametrize("cell", CELLS,
                         ids=lambda c: f"{c[0]}-{c[1]}-R{c[2]}-mu{c[3]}")
@pytest.mark.parametrize("max_add", [1, 7, 10 ** 6])
def test_device_greedy_matches_oracle(cell, max_add):
    prob, axes, R, mu = cell
    size = int(np.prod(axes))
    rng = np.random.default_rng(size + 31 * R + mu)
    code = np.sort(rng.choice(size, size=max(1, size // 60), replace=False))
    if mu > 1:
        code = np.sort(np.concatenate([code, code[: len(code) // 2]]))
    ob = OracleBackend(axes, R, prob, mu=mu)
    ob.recount(code)
    want, wdef = exact_greedy(ob, code, max_add)
    with GpuBackend(axes, R, problem=prob, mu=mu) as b:
        b.recount(code)
        got, gdef = b.greedy_fill_device(max_add)
        assert got.tolist() == want.tolist()
        assert gdef == wdef == b.uncovered()
        assert np.array_equal(b.read_cnt(), ob.cnt.astype(np.uint16))
        # the placed words joined the active multiset: they can be removed
        if len(got):
            b.ball_update(got, -1)
            ob2 = OracleBackend(axes, R, prob, mu=mu)
            ob2.recount(code)
            assert np.array_equal(b.read_cnt(), ob2.cnt.astype(np.uint16))


def test_device_greedy_covers_from_empty():
    axes, R = [3] * 8, 2
    with GpuBackend(axes, R) as b:
        b.recount(np.zeros(0, dtype=np.int64))
        placed, deficit = b.greedy_fill_device(10 ** 5)
        assert deficit == 0 and b.uncovered() == 0
        assert len(np.unique(placed)) == len(placed)
        ob = OracleBackend(axes, R)
        ob.recount(placed)
        assert ob.uncovered() == 0


def test_searcher_device_repair_lns_is_exact():
    from coldcore_b200.search import Searcher
    with GpuBackend([3] * 9, 2) as b:
        s = Searcher(b, seed=5, repair="device")
        s.build_reserve_s = s.loop_reserve_s = 0.0
        s.load([])
        s.greedy_fill(10 ** 9)
        assert s.uncov == 0 and s.verify_full() == 0
        s.peel()
        M = len(s.code) - 3
        s.ruin(3, "low")
        s.lns(M, round_budget_s=3.0, kmin=4, kmax=20, select="adaptive",
              log_every=0)
        assert s.stats["rounds"] > 0
        inc = s.uncov
        assert s.verify_full() == inc
        assert len(np.unique(s.code)) == len(s.code) <= M


@pytest.mark.parametrize("rebuild", ["0", "1"])
@pytest.mark.parametrize("cell", [("hamming", [2] * 10, 2, 1, 40),
                                  ("hamming", [5, 5, 4, 10], 1, 2, 9),
                                  ("hamming", [2] * 16, 1, 1, 3),
                                  ("hamming", [3] * 11, 1, 2, 3),
                                  ("torus_linf", [31, 33], 1, 1, 30),
                                  ("grid_linf", [25, 41], 2, 1, 30),
                                  ("lee", [4] * 5, 2, 1, 30)],
                         ids=lambda c: f"{c[0]}-{c[1]}-mu{c[3]}")
def test_device_greedy_by_updates_and_by_rebuilds(cell, rebuild, monkeypatch):
    """Gains kept by updates alone and by a transform after every placement:
    maps of just under, at and above a chunk and a block of chunks."""
    prob, axes, R, mu, steps = cell
    monkeypatch.setenv("CC_GREEDY_REBUILD", rebuild)
    size = int(np.prod(axes))
    code = np.random.default_rng(size).integers(0, size, max(1, size // 40))
    ob = OracleBackend(axes, R, prob, mu=mu)
    ob.recount(code)
    want, wdef = exact_greedy(ob, code, steps)
    with GpuBackend(axes, R, problem=prob, mu=mu) as b:
        b.recount(code)
        got, gdef = b.greedy_fill_device(steps)
        assert got.tolist() == want.tolist()
        assert gdef == wdef == b.uncovered()
        assert np.array_equal(b.read_cnt(), ob.cnt.astype(np.uint16))


@pytest.mark.parametrize("rebuild", ["0", "1", None])
@pytest.mark.parametrize("steps", [1, 5, 70])
def test_batched_greedy_by_updates_and_by_rebuilds(steps, rebuild,
                                                   monkeypatch):
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    if rebuild is not None:
        monkeypatch.setenv("CC_GREEDY_REBUILD", rebuild)
    cells = [("hamming", (3,) * 6, 2, 1), ("hamming", (4, 3, 5), 2, 2),
             ("lee", (5,) * 5, 2, 1), ("torus_linf", (5, 7, 9), 1, 1),
             ("grid_linf", (4, 5, 6), 2, 1), ("hamming", (2,) * 12, 1, 1),
             ("hamming", (2,) * 16, 2, 1), ("hamming", (6,) * 2, 2, 1)]
    with BatchEngine() as e:
        codes = []
        for p, a, R, mu in cells:
            size = int(np.prod(a))
            codes.append(np.random.default_rng(size).integers(
                0, size, 1 + size // 200))
            e.add(p, a, R, codes[-1], mu)
        e.build(48)
        for i, (p, a, R, mu) in enumerate(cells):
            e.set_table(i, wide_table(a, R, p))
        e.run()
        adds = [min(steps, 5) if np.prod(c[1]) > 4096 else steps
                for c in cells]
        got = e.greedy(np.arange(len(cells)), adds)
        for i, (p, a, R, mu) in enumerate(cells):
            ob = OracleBackend(list(a), R, p, mu=mu)
            ob.recount(codes[i])
            want, wdef = exact_greedy(ob, codes[i], adds[i])
            assert got[i][0].tolist() == want.tolist(), (i, p, a)
            assert got[i][1] == wdef
            assert np.array_equal(e.cnt(i), ob.cnt.astype(np.uint16))


def test_a_table_that_is_not_the_ball_is_never_rebuilt(monkeypatch):
    """A cell whose table lacks some of the ball's patterns: its greedy stays
    with the table's updates, whatever the rule on rebuilds says."""
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    monkeypatch.setenv("CC_GREEDY_REBUILD", "1")
    axes, R, steps = (3,) * 6, 2, 12
    size = 3 ** 6
    table = wide_table(axes, R, "hamming")
    cells = [table, table[:-7], np.concatenate([table, table[-1:]])]
    code = np.random.default_rng(8).integers(0, size, 9)
    with BatchEngine() as e:
        for _ in cells:
            e.add("hamming", axes, R, code)
        e.build(0)
        for i, tbl in enumerate(cells):
            e.set_table(i, tbl)
        e.run()
        starts = [(e.cnt(i).astype(int), e.gain(i).astype(int))
                  for i in range(len(cells))]
        got = e.greedy(np.arange(len(cells)), [steps] * len(cells))
        for i, tbl in enumerate(cells):
            cnt, gain = starts[i]
            gain[code] = -1
            strides = [3 ** j for j in range(len(axes))]
            for step, w in enumerate(got[i][0]):
                assert w == np.argmax(gain) and gain[w] > 0, (i, step)
                gain[w] = -1 << 20

                def ball(x):
                    for row in tbl:
                        y = int(x)
                        for s in row[row != 0]:
                            pw = strides[int(s) >> 24]
                            d = y // pw % 3
                            y += ((d + (int(s) & 0xFFFFFF)) % 3 - d) * pw
                        yield y
                fresh = []
                for x in ball(w):
                    if cnt[x] == 0:
                        fresh.append(x)
                    cnt[x] += 1
                for u in fresh:
                    for y in ball(u):
                        gain[y] -= 1
            assert len(got[i][0]) == steps
            assert np.array_equal(e.cnt(i), cnt.astype(np.uint16)), i


@pytest.mark.parametrize("axes,R,mu", [((2,) * 11, 1, 2), ((3,) * 11, 2, 2),
                                       ((2,) * 17, 2, 1)])
def test_batched_greedy_from_a_moved_map_is_never_rebuilt(axes, R, mu,
                                                          monkeypatch):
    """A second greedy without a step between, and a greedy after words were
    taken out: the gain map stays the last step's with the updates since, as
    it is without rebuilds, and no word is placed twice."""
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    size = int(np.prod(axes))
    code = np.random.default_rng(size).choice(size, 40, replace=False)
    got = []
    for rebuild in ("0", "1"):
        monkeypatch.setenv("CC_GREEDY_REBUILD", rebuild)
        with BatchEngine() as e:
            for _ in range(2):
                e.add("hamming", axes, R, code, mu)
            e.build(48)
            for i in range(2):
                e.set_table(i, wide_table(axes, R, "hamming"))
            e.run()
            e.update(1, code[:12], -1)
            out = e.greedy([0, 1], [6, 6]) + e.greedy([0, 1], [5, 5])
            words = np.concatenate([out[0][0], out[2][0]])
            assert len(np.unique(words)) == len(words)
            got.append([w.tolist() for w, _d in out] +
                       [e.cnt(i).tolist() for i in range(2)])
            e.run()                      # every field afresh: rebuilt again
            (w0, _), = e.greedy([0], [6])
            got[-1].append(w0.tolist())
    assert got[0] == got[1]


@pytest.mark.parametrize("axes,R,mu", [((3,) * 11, 2, 2), ((4,) * 8, 2, 2),
                                       ((2,) * 17, 3, 3)])
def test_batched_rebuilds_of_a_large_cell(axes, R, mu, monkeypatch):
    """Cells with launches of their own, mu above 1: a rebuild after every
    placement, incumbents and placed words with gains left to them."""
    from coldcore_b200.batch import BatchEngine
    from coldcore_b200.patterns import wide_table
    monkeypatch.setenv("CC_GREEDY_REBUILD", "1")
    size = int(np.prod(axes))
    code = np.random.default_rng(size).choice(size, size // 900,
                                              replace=False)
    ob = OracleBackend(list(axes), R, mu=mu)
    ob.recount(code)
    want, wdef = exact_greedy(ob, code, 6)
    with BatchEngine() as e:
        e.add("hamming", axes, R, code, mu)
        e.build(48)
        e.set_table(0, wide_table(axes, R, "hamming"))
        e.run()
        (placed, deficit), = e.greedy([0], [6])
        assert placed.tolist() == want.tolist()
        assert deficit == wdef
        assert np.array_equal(e.cnt(0), ob.cnt.astype(np.uint16))
