"""The pair form (height-0 nodes that share their pair of parents in two consecutive runs share one
pattern row) gives the oracle's results: integers bit-exact, floats within the tolerances of the
other forms, with the options of each direction, at the edges of its tiles and tables."""
import ctypes

import numpy as np
import pytest

import oracle
from tests.conftest import abs_scale, assert_matches

pytestmark = pytest.mark.gpu
DOWN, UP = 1, 2


def _pair_mode(mode):
    from grgl_gb300 import _lib

    fn = _lib.lib().grgx_debug_pair_form
    fn.restype = None
    fn.argtypes = [ctypes.c_int]
    fn(mode)


def _both(gx, g, ploidy=2, miss=None):
    """The graph again from its arrays, decided in pair form, and the oracle's."""
    a = g.export_arrays()
    kw = {} if miss is None else {"miss_node": miss}
    pg = gx.from_csr(g.num_samples, ploidy, a["down_off"], a["down_adj"], a["mut_node"], **kw).upload()
    og = oracle.OracleGraph(num_samples=g.num_samples, ploidy=ploidy, down_off=a["down_off"], down_adj=a["down_adj"],
                            mut_node=a["mut_node"], **kw)
    return pg, og


@pytest.fixture(scope="module")
def env(cuda_ok):
    import grgl_gb300 as gx

    _pair_mode(1)
    gx.set_graph_replay(False)
    try:
        # odd numbers of haplotypes (tiles of 32 and 128 end early) and of runs (a block of one run)
        g = gx.window_tree_grg(3001, 20300, seed=97)
        rng = np.random.default_rng(1)
        miss = np.full(g.num_mutations, gx.INVALID_NODE, dtype=np.uint32)
        miss[::7] = rng.integers(0, g.num_nodes, size=len(miss[::7]))
        yield (gx, *_both(gx, g, ploidy=1, miss=miss))
    finally:
        gx.set_graph_replay(True)
        _pair_mode(0)


def _rand(rng, dt, shape):
    if np.dtype(dt).kind == "f":
        return rng.standard_normal(shape).astype(dt)
    if np.dtype(dt) == np.bool_:
        return rng.integers(0, 2, size=shape).astype(bool)
    return rng.integers(0, 50, size=shape).astype(dt)


def _check(og, V, direction, got, **kw):
    rtol = 1e-12
    if V.dtype == np.float32:  # compensated float32 against the float64 product of the same inputs
        V, got = V.astype(np.float64), got.astype(np.float64)
        kw = {k: (v.astype(np.float64) if isinstance(v, np.ndarray) else v) for k, v in kw.items()}
        rtol = 1e-6
    ref = oracle.matmul(og, V, direction, **{k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in kw.items()})
    if V.dtype.kind == "f":
        assert_matches(got, ref, abs_scale(og, V, direction, kw), rtol=rtol)
    else:
        assert_matches(got, ref)


# every lane count of both element sizes, with and without a last vector or column tile in part
@pytest.mark.parametrize("dt", [np.int32, np.int64, np.uint8, np.float32, np.float64, np.bool_])
@pytest.mark.parametrize("K", [1, 2, 3, 8, 17, 33, 64, 130])
def test_pair_down_matches_oracle(env, dt, K):
    gx, g, og = env
    V = _rand(np.random.default_rng(K), dt, (K, g.num_mutations))
    _check(og, V, DOWN, gx.matmul(g, V, DOWN))


@pytest.mark.parametrize("dt", [np.int32, np.int64, np.uint8, np.float32, np.float64, np.bool_])
@pytest.mark.parametrize("K", [1, 2, 3, 8, 17, 33, 64, 130])
def test_pair_up_matches_oracle(env, dt, K):
    gx, g, og = env
    V = _rand(np.random.default_rng(K), dt, (K, g.num_samples))
    _check(og, V, UP, gx.matmul(g, V, UP))


# rows of 3, 5, 6, 9 and 10 vectors, whose lanes are no power of two (10 tiles of 3 lanes in a warp)
@pytest.mark.parametrize("dt,K", [(np.int32, 11), (np.int32, 18), (np.float32, 9), (np.float32, 20), (np.float32, 23),
                                  (np.float32, 36), (np.float32, 40), (np.float64, 5), (np.float64, 10), (np.float64, 11),
                                  (np.float64, 18), (np.float64, 20), (np.int64, 19), (np.bool_, 320)])
def test_pair_form_odd_lanes(env, dt, K):
    gx, g, og = env
    for direction, cols in ((DOWN, g.num_mutations), (UP, g.num_samples)):
        V = _rand(np.random.default_rng(K), dt, (K, cols))
        _check(og, V, direction, gx.matmul(g, V, direction))
    # as many rows as fill the ids' tiles exactly, and a few more
    for N in (128, 131, 256):
        small = gx.window_tree_grg(N, 900, seed=N)
        pg, po = _both(gx, small, ploidy=1)
        V = _rand(np.random.default_rng(N), dt, (K, pg.num_mutations))
        _check(po, V, DOWN, gx.matmul(pg, V, DOWN))


def test_pair_up_options(env):
    gx, g, og = env
    rng = np.random.default_rng(3)
    V = rng.standard_normal((5, g.num_samples))
    init = rng.standard_normal((5, g.num_nodes))
    _check(og, V, UP, gx.matmul(g, V, UP, emit_all_nodes=True, init=init), emit_all_nodes=True, init=init)
    for dt in (np.float32, np.int32):
        Vm = _rand(rng, dt, (3, g.num_samples))
        got_miss, ref_miss = (np.zeros((3, g.num_mutations), dtype=dt) for _ in range(2))
        got = gx.matmul(g, Vm, UP, by_individual=True, miss=got_miss)
        assert_matches(got, oracle.matmul(og, Vm, UP, by_individual=True, miss=ref_miss),
                       oracle.matmul(og, np.abs(Vm), UP, by_individual=True), rtol=2e-5)
        assert_matches(got_miss, ref_miss, np.full(ref_miss.shape, np.abs(Vm).sum()), rtol=2e-5)
    assert np.array_equal(gx.matmul(g, V, UP), gx.matmul(g, V, UP))


@pytest.mark.parametrize("flag", ["f32_compensated", "f64_native"])
def test_pair_down_other_accumulations(env, flag):
    gx, g, og = env
    rng = np.random.default_rng(9)
    if flag == "f64_native":
        V = rng.standard_normal((5, g.num_mutations))
        _check(og, V, DOWN, gx.matmul(g, V, DOWN, f64_native=True))
        V[0, 0], V[1, 1] = 1e300, 1e-300  # beyond the float-pair range: the FP64 path inside the same call
        _check(og, V, DOWN, gx.matmul(g, V, DOWN))
    else:
        V = rng.standard_normal((5, g.num_mutations)).astype(np.float32)
        ref = oracle.matmul(og, V.astype(np.float64), DOWN)
        got = gx.matmul(g, V, DOWN, f32_compensated=False).astype(np.float64)
        assert np.all(np.abs(got - ref) <= 2e-5 * oracle.matmul(og, np.abs(V).astype(np.float64), DOWN))


def test_pair_down_options(env):
    gx, g, og = env
    rng = np.random.default_rng(3)
    V = rng.standard_normal((5, g.num_mutations))
    init, miss = rng.standard_normal(5), rng.standard_normal((5, g.num_mutations))
    _check(og, V, DOWN, gx.matmul(g, V, DOWN, emit_all_nodes=True, init=init), emit_all_nodes=True, init=init)
    _check(og, V, DOWN, gx.matmul(g, V, DOWN, miss=miss), miss=miss)
    Vi = rng.integers(0, 9, size=(3, g.num_mutations)).astype(np.int32)
    _check(og, Vi, DOWN, gx.matmul(g, Vi, DOWN, by_individual=True), by_individual=True)
    initm = rng.standard_normal((1, g.num_nodes)).astype(np.float32)
    V1 = rng.standard_normal((1, g.num_mutations)).astype(np.float32)
    _check(og, V1, DOWN, gx.matmul(g, V1, DOWN, init=initm), init=initm)


def test_pair_down_repeats_bit_for_bit(env):
    gx, g, _ = env
    V = np.random.default_rng(4).standard_normal((20, g.num_mutations))
    assert np.array_equal(gx.matmul(g, V, DOWN), gx.matmul(g, V, DOWN))


# graphs whose runs are short, uneven or single, with nodes and haplotypes left over
@pytest.mark.parametrize("shape", ["one run", "nested", "duplicate child", "no low edges"])
def test_pair_form_other_graphs(env, shape):
    gx = env[0]
    if shape == "one run":
        N, kids = 40, {40: range(0, 20), 41: range(20, 39)}
    elif shape == "nested":  # every node conflicts with the one before it; the last haplotype has no parent
        N, kids = 33, {33: range(0, 32), 34: range(0, 16), 35: [33, 34], 36: [1, 3, 5, 35], 37: range(1, 32, 2)}
    elif shape == "duplicate child":
        N, kids = 34, {34: [0, 1, 1, 2], 35: [1, 33], 36: [3, 34, 35]}
    else:
        N, kids = 4, {4: [0, 1], 5: [4], 6: [5], 7: [6], 8: [4, 7], 9: [8]}
    n = max(kids) + 1
    off, adj = [0], []
    for v in range(n):
        adj += list(kids.get(v, []))
        off.append(len(adj))
    arrays = dict(down_off=np.array(off, dtype=np.uint64), down_adj=np.array(adj, dtype=np.uint32),
                  mut_node=np.arange(n, dtype=np.uint32))
    g = gx.from_csr(N, 1, *arrays.values())
    og = oracle.OracleGraph(num_samples=N, ploidy=1, **arrays)
    rng = np.random.default_rng(5)
    for dt in (np.int32, np.float64):
        for K in (1, 6):
            V = _rand(rng, dt, (K, n))
            _check(og, V, DOWN, gx.matmul(g, V, DOWN))
            V = _rand(rng, dt, (K, N))
            _check(og, V, UP, gx.matmul(g, V, UP))


def test_large_graph_takes_the_pair_form_by_rule(cuda_ok):
    """N=20,000, M=30,000 (6e6 edges) is over the rule's size: the same integers as without it."""
    import grgl_gb300 as gx

    g = gx.window_tree_grg(20_000, 30_000, seed=5).upload()
    V = np.random.default_rng(2).integers(0, 3, size=(6, g.num_mutations)).astype(np.int32)
    before = g.info()["device_bytes"]
    got = gx.matmul(g, V, DOWN)
    assert g.info()["device_bytes"] > before  # the form was built
    gx.set_graph_replay(False)
    _pair_mode(2)
    try:
        assert np.array_equal(got, gx.matmul(g, V, DOWN))
    finally:
        _pair_mode(0)
        gx.set_graph_replay(True)


@pytest.mark.parametrize("dt", [np.int32, np.float32, np.float64])
def test_pair_form_within_a_servers_memory(env, dt):
    """A server's batch has scratch for a part of the patterns at a time: several tables, their
    sums carried from one to the next."""
    gx, g, og = env
    with gx.Server(workers=1) as srv:
        gid = srv.add_graph(g)
        for direction, cols in ((DOWN, g.num_mutations), (UP, g.num_samples)):
            V = _rand(np.random.default_rng(6), dt, (12, cols))
            got, _ = srv.result(srv.submit(gid, V, direction), timeout=60.0)
            _check(og, V, direction, got)


@pytest.mark.parametrize("dt", [np.int32, np.int64, np.float32, np.float64])
def test_pair_up_sources_by_column_tiles(cuda_ok, dt):
    """Rows wider than L2 holds in tiles of less than a line: the last tile is partial; float64 also with
    rows that take the FP64 path."""
    import grgl_gb300 as gx

    _pair_mode(1)
    try:
        g, og = _both(gx, gx.window_tree_grg(500_002, 1_500, seed=5))
        K = 36 if np.dtype(dt).itemsize == 4 else 18  # 144 bytes a row: tiles of 64, 64 and 16
        V = _rand(np.random.default_rng(2), dt, (K, g.num_samples))
        for wide in (False, True) if dt == np.float64 else (False,):
            if wide:
                V[:, ::2] *= 1e-200
            W = V.astype(np.float64) if V.dtype.kind == "f" else V
            ref = oracle.matmul(og, W, UP)
            scale = oracle.matmul(og, np.abs(W), UP)
            assert_matches(gx.matmul(g, V, UP).astype(ref.dtype), ref, scale, rtol=1e-6 if dt == np.float32 else 1e-12)
    finally:
        _pair_mode(0)


@pytest.mark.parametrize("blocks,K", [(15, 2), (15, 7), (15, 52), (15, 56), (101, 4), (101, 8), (101, 96), (101, 100), (1, 130)])
def test_pair_down_compensated_sums(cuda_ok, blocks, K):
    """Compensated float32 over pattern rows with their error (blocks x columns up to 800, the last in tiles of
    64 columns), one at a time, and pre-summed (from 10,000): within 1e-6 of sum |terms|."""
    import grgl_gb300 as gx

    _pair_mode(1)
    try:
        g, og = _both(gx, gx.window_tree_grg(2_002, blocks * 200, seed=3))
        V = _rand(np.random.default_rng(K), np.float32, (K, g.num_mutations))
        W = V.astype(np.float64)
        assert_matches(gx.matmul(g, V, DOWN).astype(np.float64), oracle.matmul(og, W, DOWN),
                       oracle.matmul(og, np.abs(W), DOWN), rtol=1e-6)
    finally:
        _pair_mode(0)
