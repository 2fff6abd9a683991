"""Loads and stores of few columns (a thread per row): widths around the vector sizes and the last width
that takes them, with folds of a ploidy, ids through tables, missing data and initial values, on node
values kept as 4- and 8-byte numbers and as float pairs, against the oracle."""
import numpy as np
import pytest

import oracle
from tests.conftest import assert_matches

pytestmark = pytest.mark.gpu
DOWN, UP = 1, 2


@pytest.fixture(scope="module")
def env(cuda_ok):
    import grgl_gb300 as gx

    rng = np.random.default_rng(5)
    N, rows = 771, 300  # 257 individuals of ploidy 3
    adj = [np.sort(rng.choice(N, size=int(rng.integers(1, 40)), replace=False)) for _ in range(rows)]
    off = np.concatenate([np.zeros(N + 1), np.cumsum([len(a) for a in adj])]).astype(np.uint64)
    mut = rng.integers(0, N + rows, size=513).astype(np.uint32)
    miss = np.where(rng.random(513) < 0.3, rng.integers(0, N + rows, size=513), 0x7fffffff).astype(np.uint32)
    arrays = dict(down_off=off, down_adj=np.concatenate(adj).astype(np.uint32), mut_node=mut, miss_node=miss)
    return gx, gx.from_csr(N, 3, *arrays.values()).upload(), oracle.OracleGraph(num_samples=N, ploidy=3, **arrays)


@pytest.mark.parametrize("dt", [np.int8, np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 6, 7, 12, 13])
@pytest.mark.parametrize("wide", [False, True])
def test_narrow_loads_and_stores(env, dt, K, wide):
    """float64 with `wide` spans more binades than float pairs carry."""
    gx, g, og = env
    rng = np.random.default_rng(K)
    isf = np.dtype(dt).kind == "f"

    def values(*shape):
        v = rng.standard_normal(shape) if isf else rng.integers(-3, 4, size=shape)
        if wide and dt == np.float64:
            v[..., ::2] *= 1e-200
        return v.astype(dt)

    eps = 1e-6 if dt == np.float32 else 1e-12
    up = np.float64 if isf else dt  # the oracle's type
    for direction, cols in ((UP, 771), (DOWN, 513)):
        for kw in ({}, {"emit_all_nodes": True}, {"by_individual": True}):
            ind = "by_individual" in kw
            V = values(K, 257 if ind and direction == UP else cols)
            init = None if ind else values(K, g.num_nodes)
            miss = None if "emit_all_nodes" in kw else values(K, 513)

            def run(f, to, change=lambda v: v):
                v, i, m = (None if x is None else change(x).astype(to) for x in (V, init, miss))
                return f(v, i, m), m

            call = dict(direction=direction, **kw)
            got = run(lambda v, i, m: gx.matmul(g, v, init=i, miss=m, **call), dt)
            ref, top = (run(lambda v, i, m: oracle.matmul(og, v, init=i, miss=m, **call), up, c)
                        for c in (lambda v: v, np.abs))
            for a, b, s in zip(got, ref, top):
                if a is not None:
                    assert_matches(a.astype(up), b, s, rtol=eps)


@pytest.mark.parametrize("dt", [np.int8, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("K,rows", [(20, 60000), (20, 59999), (21, 60000)])
def test_last_sizes_of_narrow_loads_and_stores(cuda_ok, dt, K, rows):
    """Every sample carries one mutation, in an order that is its own inverse: both products move columns."""
    import grgl_gb300 as gx

    order = np.arange(rows, dtype=np.uint32) ^ 1 if rows % 2 == 0 else np.arange(rows, dtype=np.uint32)[::-1].copy()
    g = gx.from_csr(rows, 1, np.zeros(rows + 1, dtype=np.uint64), np.zeros(0, dtype=np.uint32), order).upload()
    V = np.arange(K * rows).reshape(K, rows).astype(dt)
    for direction in (UP, DOWN):
        assert np.array_equal(gx.matmul(g, V, direction), V[:, order])
