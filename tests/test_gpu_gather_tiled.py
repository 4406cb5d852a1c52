"""The tiled gather (a block walks a tile of the support table for a group
of candidates), with and without the predicate bit plane, against the
oracle and against the per-word walk, for Hamming, Lee, torus and
mixed-radix cells, mu = 1 and 2, every role."""
import numpy as np
import pytest

from coldcore_b200.gpu import GpuBackend
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
