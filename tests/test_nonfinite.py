"""Infinities and NaN in the input reach exactly the outputs whose sums have such a term, in the pair form, the
lists of single columns, levels of short rows and chains of small levels: finite outputs stay right."""
import numpy as np
import pytest

import oracle
from tests.test_pair_form import DOWN, UP, _both, _pair_mode

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["pair", "levels"])
def env(cuda_ok, request):
    import grgl_gb300 as gx

    _pair_mode(1 if request.param == "pair" else 2)
    try:
        yield (gx, *_both(gx, gx.window_tree_grg(3001, 8100, seed=11), ploidy=1))
    finally:
        _pair_mode(0)


@pytest.mark.parametrize("K", [1, 2, 5, 24, 70])
@pytest.mark.parametrize("dt,kw", [(np.float32, {}), (np.float32, {"f32_compensated": False}), (np.float64, {}),
                                   (np.float64, {"f64_native": True})])
@pytest.mark.parametrize("direction", [DOWN, UP])
def test_nonfinite_inputs(env, K, dt, kw, direction):
    gx, g, og = env
    rng = np.random.default_rng(K)
    V = rng.standard_normal((K, g.num_samples if direction == UP else g.num_mutations)).astype(dt)
    clean = V.copy()
    for value in (np.inf, -np.inf, np.nan):
        V[rng.integers(0, K), rng.integers(0, V.shape[1])] = value
    touched = np.where(np.isfinite(V), 0, 1).astype(np.int32)
    touched = oracle.matmul(og, touched, direction) > 0
    scale = oracle.matmul(og, np.abs(clean).astype(np.float64), direction)
    ref = oracle.matmul(og, clean.astype(np.float64), direction)
    for replay in (False, True):
        gx.set_graph_replay(replay)
        try:
            got = gx.matmul(g, V, direction, **kw)
        finally:
            gx.set_graph_replay(True)
        assert not np.any(np.isfinite(got[touched]))
        rest = ~touched
        tol = 2e-5 if kw.get("f32_compensated") is False else 1e-6 if dt == np.float32 else 1e-12
        assert np.all(np.abs(got[rest] - ref[rest]) <= tol * scale[rest])
