"""The life of a graph's pair form (pair_plan.h): what the first call of each direction builds and what it
leaves alone, on several threads, and where it cannot be built."""
import ctypes
import threading

import numpy as np
import pytest

from tests.test_pair_form import DOWN, UP, _both, _check, _pair_mode, _rand

pytestmark = pytest.mark.gpu


@pytest.fixture()
def env(cuda_ok):
    import grgl_gb300 as gx

    _pair_mode(1)
    gx.set_graph_replay(False)
    try:
        yield (gx, *_both(gx, gx.window_tree_grg(3001, 20300, seed=97), ploidy=1))
    finally:
        gx.set_graph_replay(True)
        _pair_mode(0)


def _analysis(g):
    from grgl_gb300 import _lib

    out = ctypes.c_void_p()
    _lib.check(_lib.lib().grgx_debug_pair_analysis(g._h, ctypes.byref(out)))
    return out.value


def _input(g, direction, dt, K, seed=0):
    return _rand(np.random.default_rng(seed), dt, (K, g.num_samples if direction == UP else g.num_mutations))


@pytest.mark.parametrize("first", [DOWN, UP])
def test_second_direction_leaves_the_analysis_in_place(env, first):
    """Calls of the first direction read it without the graph's lock."""
    gx, g, og = env
    gx.matmul(g, _input(g, first, np.int32, 6), first)
    before = _analysis(g)
    assert before
    V = _input(g, 3 - first, np.int32, 6)
    _check(og, V, 3 - first, gx.matmul(g, V, 3 - first))
    assert _analysis(g) == before


@pytest.mark.parametrize("first", [DOWN, UP])
def test_first_calls_of_both_directions_on_several_threads(env, first):
    """Products of one direction run while another thread's first call builds the other."""
    gx, g, og = env
    gx.matmul(g, _input(g, first, np.float64, 3), first)  # this direction is built
    started, errs = threading.Event(), []

    def work(i):
        try:
            for k in range(6):
                d = first if i else 3 - first
                V = _input(g, d, (np.int32, np.float64)[i % 2], 3 + i, seed=10 * i + k)
                if i:
                    started.set()
                else:
                    started.wait()
                _check(og, V, d, gx.matmul(g, V, d))
        except Exception as e:  # reported below
            errs.append(e)
            started.set()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errs, errs


def _refuse(skip, count):
    """Fails `count` allocations of plan memory after `skip` more; returns how many have failed since the last call."""
    from grgl_gb300 import _lib

    fn = _lib.lib().grgx_debug_plan_alloc
    fn.restype = ctypes.c_longlong
    fn.argtypes = [ctypes.c_longlong, ctypes.c_longlong]
    return fn(skip, count)


def _built(g, direction):
    from grgl_gb300 import _lib

    out = (ctypes.c_uint64 * 4)()
    _lib.check(_lib.lib().grgx_debug_pair_counts(g._h, direction, out))
    return out[1] > 0


@pytest.mark.parametrize("second", [False, True])
@pytest.mark.parametrize("direction", [DOWN, UP])
def test_out_of_memory_in_a_build(env, direction, second):
    """Every allocation of a build fails in turn: once, and the build is made again; then for good, and calls of
    the direction take the other forms, without building again or keeping memory."""
    gx, g, og = env
    V, W = (_input(g, d, np.int32, 6) for d in (direction, 3 - direction))
    a = g.export_arrays()
    skip, failed, kept = 0, True, set()
    while failed:
        for count in (1, 1 << 40):
            h = gx.from_csr(g.num_samples, 1, a["down_off"], a["down_adj"], a["mut_node"]).upload()
            if second:
                gx.matmul(h, W, 3 - direction)
            bytes0 = h.info()["device_bytes"]
            try:
                _refuse(skip, count)
                _check(og, V, direction, gx.matmul(h, V, direction))
                failed = _refuse(skip, count)
                assert failed <= 2
                assert _built(h, direction) == (failed < 2)
                if failed == 2:
                    kept.add(h.info()["device_bytes"] - bytes0)
                _check(og, V, direction, gx.matmul(h, V, direction))
                assert _refuse(-1, 0) == 0
            finally:
                _refuse(-1, 0)
            _check(og, W, 3 - direction, gx.matmul(h, W, 3 - direction))
            assert _built(h, 3 - direction)
        skip += 1
    # (the UP edges between inner nodes, once complete, serve the split form too)
    assert skip > 10 and 0 in kept and len(kept) == (1 if direction == DOWN else 2)


@pytest.mark.parametrize("first", [DOWN, UP])
def test_more_table_rows_than_lists_can_number(env, first):
    """UP takes another form then; DOWN, whose patterns have no such rows, keeps the pair form."""
    from grgl_gb300 import _lib

    gx, g, og = env
    fn = _lib.lib().grgx_debug_pair_rows
    fn.restype = None
    fn.argtypes = [ctypes.c_longlong]
    fn(1000)
    try:
        for direction in (first, 3 - first):
            V = _input(g, direction, np.int32, 6)
            _check(og, V, direction, gx.matmul(g, V, direction))
            assert _built(g, direction) == (direction == DOWN)
    finally:
        fn(0x3fffffff)


def _form(g, dt, K, direction, pair=-1):
    """The form a call takes; `pair` 0 or 1: with that measured choice recorded."""
    from grgl_gb300 import _lib
    from grgl_gb300.api import _DTYPE_CODES

    out = ctypes.c_int()
    fn = _lib.lib().grgx_debug_call_form
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.c_uint32, ctypes.c_int,
                   ctypes.POINTER(ctypes.c_int)]
    _lib.check(fn(g._h, _DTYPE_CODES[np.dtype(dt)], K, direction, 0, pair, ctypes.byref(out)))
    return ("unsplit", "in split form", "in pair form")[out.value]


@pytest.mark.parametrize("direction", [DOWN, UP])
def test_autotune_chooses_among_all_forms(cuda_ok, direction):
    """The form it reports is the one that calls take, also against the rules, and results hold in any."""
    import grgl_gb300 as gx

    g = gx.window_tree_grg(40_000, 9_000, seed=5).upload()  # 3.6e6 edges, two blocks of samples
    try:
        for dt, K in ((np.int32, 6), (np.int32, 1), (np.float32, 9), (np.float64, 20)):
            V = _input(g, direction, dt, K)
            exact = gx.matmul(g, V.astype(np.float64), direction, f64_native=True)
            by_rule = _form(g, dt, K, direction)
            report = gx.autotune(g, dt, K, direction)
            form = _form(g, dt, K, direction)
            assert report.splitlines()[-1].endswith(f"runs {form} for this shape")
            assert ("pair sweep" in report) == (by_rule == "in pair form")
            for pair in (0, 1):
                assert (_form(g, dt, K, direction, pair) == "in pair form") == (pair == 1 and by_rule == "in pair form")
                gx.set_graph_replay(False)
                got = gx.matmul(g, V, direction)
                gx.set_graph_replay(True)
                scale = gx.matmul(g, np.abs(V).astype(np.float64), direction, f64_native=True)
                assert np.all(np.abs(got - exact) <= {4: 1e-6, 8: 1e-12}[V.itemsize] * scale)
            report = gx.autotune(g, dt, K, direction)  # (measured again, whatever was recorded)
            assert report.splitlines()[-1].endswith(f"runs {_form(g, dt, K, direction)} for this shape")
    finally:
        gx.autotune_clear()
        gx.set_graph_replay(True)


@pytest.mark.parametrize("N,M", [(3001, 20300), (128, 900), (131, 900), (256, 900), (2002, 200), (2002, 20200)])
def test_graphs_of_the_form_tests_take_it(env, N, M):
    """The oracle comparisons of the pair form (test_pair_form.py) are of that form."""
    gx = env[0]
    g, og = _both(gx, gx.window_tree_grg(N, M, seed=N), ploidy=1)
    for direction in (DOWN, UP):
        for dt, K in ((np.int32, 2), (np.float32, 33), (np.float64, 1)):
            V = _input(g, direction, dt, K)
            _check(og, V, direction, gx.matmul(g, V, direction))
            assert _form(g, dt, K, direction) == "in pair form" and _built(g, direction)


def test_duplicate_children_take_another_form(env):
    """A height-0 node that is the same node's child twice has no single pattern."""
    import oracle

    gx = env[0]
    arrays = dict(down_off=np.array([0] * 35 + [4, 6, 9], dtype=np.uint64),
                  down_adj=np.array([0, 1, 1, 2, 1, 33, 3, 34, 35], dtype=np.uint32), mut_node=np.arange(37, dtype=np.uint32))
    g, og = gx.from_csr(34, 1, *arrays.values()), oracle.OracleGraph(num_samples=34, ploidy=1, **arrays)
    for direction in (DOWN, UP):
        V = _input(g, direction, np.int32, 2)
        _check(og, V, direction, gx.matmul(g, V, direction))
        assert _form(g, np.int32, 2, direction) == "unsplit" and not _built(g, direction)


def _ranges(g, dt, K, direction, limit):
    from grgl_gb300 import _lib
    from grgl_gb300.api import _DTYPE_CODES

    out = ctypes.c_int()
    fn = _lib.lib().grgx_debug_pair_ranges
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.c_uint32, ctypes.c_uint64,
                   ctypes.POINTER(ctypes.c_int)]
    _lib.check(fn(g._h, _DTYPE_CODES[np.dtype(dt)], K, direction, 0, limit, ctypes.byref(out)))
    return out.value


@pytest.fixture(scope="module")
def many_blocks(cuda_ok):
    """300 blocks: five segments of UP lists."""
    import grgl_gb300 as gx

    _pair_mode(1)
    try:
        yield _both(gx, gx.window_tree_grg(2002, 60_000, seed=3), ploidy=1)
    finally:
        _pair_mode(0)


# kinds with state between UP's tables and levels, and without; columns in one tile and several
@pytest.mark.parametrize("dt,K", [(np.int32, 12), (np.int64, 3), (np.float32, 40), (np.float64, 1), (np.float64, 18), (np.bool_, 70)])
@pytest.mark.parametrize("direction", [DOWN, UP])
def test_several_tables(env, many_blocks, direction, dt, K):
    """With little scratch the patterns' rows are made in parts, whose sums are carried on."""
    gx, (g, og) = env[0], many_blocks
    V = _input(g, direction, dt, K)
    seen = set()
    try:
        for shift in range(40, 11, -1):
            for limit in (1 << shift, 3 << (shift - 2)):
                n = _ranges(g, dt, K, direction, limit)
                if n not in seen:
                    seen.add(n)
                    _check(og, V, direction, gx.matmul(g, V, direction))
    finally:
        _ranges(g, dt, K, direction, 0)
    assert {0, 1, 2} <= seen and max(seen) >= 3, seen


@pytest.mark.parametrize("direction", [DOWN, UP])
def test_first_call_inside_an_applications_capture(env, direction):
    """It takes a form that needs no build, and a later call the pair form; the captured graph stays right."""
    import torch

    gx, g, og = env
    V = _input(g, direction, np.float64, 6)
    x = torch.zeros(V.shape, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = gx.matmul(g, x, direction)
    assert not _built(g, direction)
    x.copy_(torch.from_numpy(V))
    graph.replay()
    _check(og, V, direction, out.cpu().numpy())
    _check(og, V, direction, gx.matmul(g, V, direction))
    assert _built(g, direction)
    graph.replay()
    _check(og, V, direction, out.cpu().numpy())
    del graph


@pytest.mark.parametrize("direction", [DOWN, UP])
def test_build_beside_an_applications_capture(env, direction):
    """A first call on another thread, while this one captures."""
    import torch

    gx, g, og = env
    V = _input(g, direction, np.int32, 6)
    got = []
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x + 1
        t = threading.Thread(target=lambda: got.append(_form(g, np.int32, 6, direction)))
        t.start()
        t.join()
        z = y * 2
    graph.replay()
    assert got == ["in pair form"] and float(z.sum()) == 4000.0
    _check(og, V, direction, gx.matmul(g, V, direction))
