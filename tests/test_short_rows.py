"""Levels of short rows (one group of lanes per row): rows of 0 to 128 edges around the kernel's batch
of four and the float-pair run of 32, next to a level that is too long for it, in both directions,
against the oracle: integers bit-exact, floats within the usual tolerances."""
import numpy as np
import pytest

import oracle
from tests.conftest import assert_matches_oracle

pytestmark = pytest.mark.gpu
DOWN, UP = 1, 2


@pytest.fixture(scope="module")
def env(cuda_ok):
    import grgl_gb300 as gx

    rng = np.random.default_rng(8)
    N = 700
    degrees = [1] * 400 + [2, 3, 4, 5, 8, 28, 29, 31, 32, 33, 64, 100, 128] + [1, 4] * 100
    off, adj = [0] * (N + 1), []
    layer = range(N)
    for last in (False, False, True):  # two short levels, then one with a row past the longest
        start = len(off) - 1
        for d in degrees + ([129] if last else []):
            adj += sorted(rng.choice(np.array(layer), size=d, replace=False).tolist())
            off.append(len(adj))
        layer = range(start, len(off) - 1)
    n = len(off) - 1
    arrays = dict(down_off=np.array(off, dtype=np.uint64), down_adj=np.array(adj, dtype=np.uint32),
                  mut_node=rng.integers(0, n, size=2 * n).astype(np.uint32))
    return gx, gx.from_csr(N, 1, *arrays.values()).upload(), oracle.OracleGraph(num_samples=N, ploidy=1, **arrays)


@pytest.mark.parametrize("dt", [np.int32, np.int64, np.float32, np.float64, np.bool_])
@pytest.mark.parametrize("K", [1, 2, 5, 40, 130])
@pytest.mark.parametrize("direction", [UP, DOWN])
def test_short_levels_match_oracle(env, dt, K, direction):
    gx, g, og = env
    rng = np.random.default_rng(K)
    shape = (K, g.num_samples if direction == UP else g.num_mutations)
    V = rng.standard_normal(shape).astype(dt) if np.dtype(dt).kind == "f" else rng.integers(0, 2, size=shape).astype(dt)
    assert_matches_oracle(og, V, direction, gx.matmul(g, V, direction))


def test_short_levels_with_initial_values(env):
    gx, g, og = env
    rng = np.random.default_rng(3)
    V, init = rng.standard_normal((6, g.num_samples)), rng.standard_normal((6, g.num_nodes))
    got = gx.matmul(g, V, UP, emit_all_nodes=True, init=init)
    ref = oracle.matmul(og, V, UP, emit_all_nodes=True, init=init)
    scale = oracle.matmul(og, np.abs(V), UP, emit_all_nodes=True, init=np.abs(init))
    assert np.all(np.abs(got - ref) <= 1e-12 * scale)
