"""Window passes over two axes at a time against the oracle: torus and open
grid, odd and ragged axes, two to four of them, windows in and above the
pair form's range, mu = 1 and 2, repeated codewords."""
import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
from oracle.dp_oracle import OracleBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problem", ["torus_linf", "grid_linf"])
@pytest.mark.parametrize("axes,R,mu", [
    ([40, 33], 1, 1), ([33, 257], 2, 2), ([17, 18, 19], 1, 1),
    ([7, 20, 9], 3, 1), ([19, 5, 6, 7], 2, 2), ([21, 23], 4, 1),
    ([300, 3], 1, 1), ([3, 301], 1, 2), ([18], 2, 1), ([512, 512], 1, 1)])
def test_paired_window_passes_match_the_oracle(problem, axes, R, mu):
    if problem == "torus_linf" and min(axes) < 2 * R + 1:
        pytest.skip("the torus window must fit its axis")
    size = int(np.prod(axes))
    rng = np.random.default_rng(size + R)
    code = rng.integers(0, size, size=max(3, size // 30))
    code = np.concatenate([code, code[:2]])
    o = OracleBackend(axes, R, problem=problem, mu=mu)
    o.recount(code)
    with GpuBackend(axes, R, problem=problem, mu=mu) as b:
        b.recount(code)
        assert np.array_equal(b.read_cnt(), o.read_cnt())
        assert b.uncovered() == o.uncovered()
        for field in ("gain_map", "loss_map", "gain_map"):
            getattr(b, field)()
            getattr(o, field)()
            assert np.array_equal(b.map_all(), o.map), field
        assert sum(int(r[1]) for r in b.plan(1, 1)) == len(axes)
