"""Chains of small levels in one launch (chain.cuh): graphs of 2 to 40 levels with rows of 1 to 512
edges, below and above the sizes that chains take, against the oracle, and the same with CUDA-graph
replay."""
import numpy as np
import pytest

import oracle
from tests.conftest import assert_matches_oracle

pytestmark = pytest.mark.gpu
DOWN, UP = 1, 2


def _graph(gx, levels, width, longest, N=600):
    """`levels` levels of `width` rows; every row has a child in the level below, some `longest`."""
    rng = np.random.default_rng(levels)
    off, adj = [0] * (N + 1), []
    below = np.arange(N)
    for _ in range(levels):
        first = len(off) - 1
        for r in range(width):
            d = longest if r == 0 else int(rng.integers(0, 12))
            kids = np.concatenate([rng.choice(below, size=1), rng.choice(first, size=min(d, first - 1), replace=False)])
            adj.append(np.unique(kids))
            off.append(off[-1] + len(adj[-1]))
        below = np.arange(first, len(off) - 1)
    n = len(off) - 1
    arrays = dict(down_off=np.array(off, dtype=np.uint64), down_adj=np.concatenate(adj).astype(np.uint32),
                  mut_node=rng.integers(0, n, size=n + 50).astype(np.uint32))
    return gx.from_csr(N, 1, *arrays.values()).upload(), oracle.OracleGraph(num_samples=N, ploidy=1, **arrays)


@pytest.fixture(scope="module", params=[(2, 300, 512), (12, 40, 200), (40, 15, 3), (5, 2500, 513), (3, 6000, 31)])
def env(cuda_ok, request):
    import grgl_gb300 as gx

    return (gx, *_graph(gx, *request.param))


@pytest.mark.parametrize("dt", [np.int32, np.int64, np.float32, np.float64, np.bool_])
@pytest.mark.parametrize("K", [1, 2, 6, 40])
def test_chains_match_oracle(env, dt, K):
    gx, g, og = env
    rng = np.random.default_rng(K)
    for direction, cols in ((UP, g.num_samples), (DOWN, g.num_mutations)):
        V = (rng.standard_normal((K, cols)) if np.dtype(dt).kind == "f" else rng.integers(0, 2, size=(K, cols))).astype(dt)
        for replay in (False, True):
            gx.set_graph_replay(replay)
            try:
                assert_matches_oracle(og, V, direction, gx.matmul(g, V, direction))
            finally:
                gx.set_graph_replay(True)


def test_chains_take_the_fp64_path_and_initial_values(env):
    gx, g, og = env
    rng = np.random.default_rng(7)
    V = rng.standard_normal((2, g.num_samples))
    V[0, 0], V[1, 1] = 1e300, 1e-300
    assert_matches_oracle(og, V, UP, gx.matmul(g, V, UP))
    W, init = rng.integers(0, 9, size=(3, g.num_mutations)).astype(np.int32), np.arange(3, dtype=np.int32)
    assert np.array_equal(gx.matmul(g, W, DOWN, emit_all_nodes=True, init=init),
                          oracle.matmul(og, W, DOWN, emit_all_nodes=True, init=init))
