"""Single 4-byte columns in split form (staged.cu): lists of every length around a load of 8 ids, a
step of 64 and a piece of 1,024, starting at every offset to a load's boundary, against the oracle."""
import ctypes

import numpy as np
import pytest

import oracle
from tests.conftest import assert_matches_oracle

pytestmark = pytest.mark.gpu
DOWN, UP = 1, 2


@pytest.fixture(scope="module", params=[1024, 32768])
def env(cuda_ok, request):
    import grgl_gb300 as gx
    from grgl_gb300 import _lib

    split, forms = _lib.lib().grgx_debug_up_split, _lib.lib().grgx_debug_split_forms
    split.restype = forms.restype = None
    split.argtypes = [ctypes.c_longlong, ctypes.c_ulonglong]
    forms.argtypes = [ctypes.c_int, ctypes.c_int]
    split(request.param, 0)
    forms(1, 1)
    gx.set_graph_replay(False)
    try:
        rng = np.random.default_rng(3)
        N = 2 * request.param + 5  # a last block of five
        degrees = [1, 2, 7, 8, 9, 63, 64, 65, 71, 72, 127, 128, 129, 500, 1023, 1024] * 3 + [N // 2, N - 1, N] + [3] * 40
        degrees += [11] * (2 * request.param // 1000)
        off, adj = [0] * (N + 1), []
        for d in degrees:
            adj.append(np.sort(rng.choice(N, size=d, replace=False)))
            off.append(off[-1] + d)
        low = len(off) - 1
        for _ in range(max(1000, request.param + 100)):  # parents enough for two blocks of them
            adj.append(np.sort(np.concatenate([rng.choice(N, size=2, replace=False), rng.integers(N, low, size=1)])))
            off.append(off[-1] + 3)
        n = len(off) - 1
        arrays = dict(down_off=np.array(off, dtype=np.uint64), down_adj=np.concatenate(adj).astype(np.uint32),
                      mut_node=rng.integers(0, n, size=n).astype(np.uint32))
        yield gx, gx.from_csr(N, 1, *arrays.values()).upload(), oracle.OracleGraph(num_samples=N, ploidy=1, **arrays)
    finally:
        gx.set_graph_replay(True)
        split(32768, 64 << 20)
        forms(0, 1)


@pytest.mark.parametrize("dt", [np.int32, np.uint8, np.float32, np.bool_])
@pytest.mark.parametrize("direction", [UP, DOWN])
def test_staged_lists_match_oracle(env, dt, direction):
    gx, g, og = env
    rng = np.random.default_rng(1)
    for K in ((1, 31) if dt == np.bool_ else (1,)):
        shape = (K, g.num_samples if direction == UP else g.num_mutations)
        V = rng.standard_normal(shape).astype(dt) if dt == np.float32 else rng.integers(0, 2, size=shape).astype(dt)
        got = gx.matmul(g, V, direction)
        assert_matches_oracle(og, V, direction, got)
        assert np.array_equal(got, gx.matmul(g, V, direction))


def test_staged_plain_float32(env):
    gx, g, og = env
    for direction, cols in ((UP, g.num_samples), (DOWN, g.num_mutations)):
        V = np.random.default_rng(2).standard_normal((1, cols)).astype(np.float32)
        ref = oracle.matmul(og, V.astype(np.float64), direction)
        scale = oracle.matmul(og, np.abs(V).astype(np.float64), direction)
        assert np.all(np.abs(gx.matmul(g, V, direction, f32_compensated=False) - ref) <= 2e-5 * scale)


def test_staged_with_initial_values(env):
    gx, g, og = env
    rng = np.random.default_rng(4)
    V, init = rng.integers(0, 9, size=(1, g.num_samples)).astype(np.int32), np.array([7], dtype=np.int32)
    assert np.array_equal(gx.matmul(g, V, UP, emit_all_nodes=True, init=init),
                          oracle.matmul(og, V, UP, emit_all_nodes=True, init=init))
