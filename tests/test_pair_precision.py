"""Compensated float32 in pair form is at least as near to the float64 product as the sweep over edges, which
the pair form takes the place of: the norm of the error over all outputs, plain and standardized products."""
import numpy as np
import pytest

from tests.test_pair_form import DOWN, UP, _pair_mode

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs(cuda_ok):
    import grgl_gb300 as gx

    made = {}

    def get(N, M):
        if (N, M) not in made:
            made.clear()
            made[N, M] = gx.window_tree_grg(N, M, seed=42).upload()
        return made[N, M]

    gx.set_graph_replay(False)
    try:
        yield gx, get
    finally:
        gx.set_graph_replay(True)
        _pair_mode(0)


# blocks x columns of every kind of DOWN sum (pair_run.cu), and the narrow and wide ends of UP
@pytest.mark.parametrize("N,M,direction,K", [
    (20_000, 250_000, DOWN, 6), (20_000, 250_000, DOWN, 9), (20_000, 250_000, DOWN, 12), (20_000, 250_000, DOWN, 24),
    (20_000, 250_000, UP, 2), (20_000, 250_000, UP, 6), (20_000, 250_000, UP, 33),
    (100_000, 20_000, DOWN, 12), (100_000, 20_000, DOWN, 100), (200_000, 3_000, DOWN, 48), (200_000, 3_000, DOWN, 64)])
@pytest.mark.parametrize("standardized", [False, True])
def test_errors_at_or_below_the_sweeps(graphs, N, M, direction, K, standardized):
    import torch

    gx, get = graphs
    g = get(N, M)
    product = gx.matmul_standardized if standardized else gx.matmul

    def error(mode, x, exact):
        _pair_mode(mode)
        got = product(g, x, direction).double()
        return float((got - exact).square().sum()), float(exact.square().sum())

    total = {1: 0.0, 2: 0.0}
    for seed in range(4):
        torch.manual_seed(seed)
        x = torch.randn((K, g.num_samples if direction == UP else g.num_mutations), device="cuda")
        _pair_mode(2)
        exact = product(g, x.double(), direction, f64_native=True)
        for mode in total:
            e, n = error(mode, x, exact)
            total[mode] += e / n
    assert total[1] <= total[2], (np.sqrt(total[1] / 4), np.sqrt(total[2] / 4))


# (short rows, whose sums take runs of four pattern rows; many blocks; few and many columns)
@pytest.mark.parametrize("N,M,direction,K", [
    (20_000, 50_000, DOWN, 1), (20_000, 50_000, DOWN, 3), (20_000, 50_000, DOWN, 9), (20_000, 50_000, DOWN, 64),
    (20_000, 50_000, UP, 1), (20_000, 50_000, UP, 6), (20_000, 50_000, UP, 33),
    (100_000, 20_000, DOWN, 2), (100_000, 20_000, DOWN, 18), (200_000, 3_000, DOWN, 2), (200_000, 3_000, DOWN, 6)])
@pytest.mark.parametrize("inputs", ["normal", "positive", "standardized"])
def test_float64_errors_at_or_below_the_sweeps(graphs, N, M, direction, K, inputs):
    import torch

    gx, get = graphs
    g = get(N, M)
    product = gx.matmul_standardized if inputs == "standardized" else gx.matmul
    total = {1: 0.0, 2: 0.0}
    for seed in range(4):
        torch.manual_seed(seed)
        x = torch.randn((K, g.num_samples if direction == UP else g.num_mutations), device="cuda", dtype=torch.float64)
        if inputs == "positive":
            x = x.abs()
        _pair_mode(2)
        exact = product(g, x, direction, f64_native=True)
        for mode in total:
            _pair_mode(mode)
            total[mode] += float((product(g, x, direction) - exact).square().sum() / exact.square().sum())
    assert total[1] <= total[2], (np.sqrt(total[1] / 4), np.sqrt(total[2] / 4))


@pytest.mark.parametrize("N,M,direction,K", [
    (20_000, 50_000, DOWN, 2), (20_000, 50_000, DOWN, 18), (20_000, 50_000, UP, 2), (20_000, 50_000, UP, 18),
    (100_000, 20_000, DOWN, 3), (100_000, 20_000, DOWN, 33), (100_000, 20_000, UP, 9), (100_000, 20_000, UP, 64)])
def test_plain_sums_near_the_sweeps(graphs, N, M, direction, K):
    """Plain float32 and FP64 sums of one lane per row, grouped: within 1.25 times the sweep's error (whose terms are
    spread over lanes), where sums one by one have up to three times it.  FP64's error is taken against inputs in
    two halves whose sums are exact."""
    import torch

    gx, get = graphs
    g = get(N, M)
    total = {(m, dt): 0.0 for m in (1, 2) for dt in (torch.float32, torch.float64)}
    for seed in range(4):
        torch.manual_seed(seed)
        x = torch.randn((K, g.num_samples if direction == UP else g.num_mutations), device="cuda", dtype=torch.float64)
        high = (x * 2**22).round() / 2**22
        low = ((x - high) * 2**48).round() / 2**48
        _pair_mode(2)
        H, L = (gx.matmul(g, v, direction, f64_native=True) for v in (high, low))
        x32 = x.float()
        exact32 = gx.matmul(g, x32.double(), direction, f64_native=True)
        for mode in (1, 2):
            _pair_mode(mode)
            e = (gx.matmul(g, high + low, direction, f64_native=True) - H) - L
            total[mode, torch.float64] += float(e.square().sum() / H.square().sum())
            e = gx.matmul(g, x32, direction, f32_compensated=False).double() - exact32
            total[mode, torch.float32] += float(e.square().sum() / exact32.square().sum())
    for dt in (torch.float32, torch.float64):
        assert total[1, dt] <= 1.25**2 * total[2, dt], (dt, np.sqrt(total[1, dt] / 4), np.sqrt(total[2, dt] / 4))


def test_plain_sums_of_short_rows(cuda_ok):
    """Rows of eight edges, one group of lanes each, four edges at a time as a tree.  The same sums of N(0,1) values in
    numpy leave 0.80 u of the norm as trees of four and 0.94 u one by one (u = 2^-24): the line lies between."""
    import torch

    import grgl_gb300 as gx

    rng = np.random.default_rng(4)
    N, rows, d = 3000, 12000, 8
    adj = np.sort(np.stack([rng.choice(N, size=d, replace=False) for _ in range(rows)])).astype(np.uint32)
    off = np.concatenate([np.zeros(N, dtype=np.uint64), np.arange(rows + 1, dtype=np.uint64) * d])
    g = gx.from_csr(N, 1, off, adj.ravel(), np.arange(N, N + rows, dtype=np.uint32)).upload()
    x = torch.from_numpy(rng.standard_normal((8, N)).astype(np.float32)).cuda()
    exact = x.double()[:, torch.from_numpy(adj.astype(np.int64)).cuda()].sum(-1)
    got = gx.matmul(g, x, UP, f32_compensated=False).double()
    assert float((got - exact).norm() / exact.norm()) <= 0.87 * 2.0**-24
