"""GPU: the float32 forms of retention and differential attention at the edges of their tiles, against the float64 oracle: heads up to the
register limits and one above, portions around 16 tokens, 16 queries and 32 keys, value sizes of one and two column groups."""
import pytest
import torch

from test_gpu_fabezen_kernels import DeltaCase
from test_gpu_hybrid_kernels import BF, F32, Case, X, err, ret_case, run_ret  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,dv,dims", [(2, 64, 16, 64), (1, 65, 17, 6), (2, 128, 256, 128), (1, 129, 15, 128), (2, 256, 40, 0), (1, 257, 33, 254)])
@pytest.mark.parametrize("dt", [BF, F32])
def test_retention_row_groups(X, H, d, dv, dims, dt):      # noqa: F811
    T = 50
    case = ret_case(X, T, H, d, dv, dims, dt)
    for cuts in ([T], [16, 17, 1, 15, 1], [31, 19]):
        o, S = run_ret(X, case, H, d, dv, dims, cuts, 1)
        assert err(o, case[1][0]) < 2e-5 and err(S, case[1][1]) < 2e-5


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 128), (2, 2, 4, 4), (3, 1, 36, 132), (2, 1, 128, 256), (1, 1, 12, 260), (4, 2, 66, 128)])
def test_differential_attention_tiles(X, scmx, H, G, d, dv):      # noqa: F811
    T = 150
    c = Case(scmx, T, H, G, d, dv, F32)
    c.fill()
    want = c.want(list(range(T)))
    for lo, hi in ((0, T), (0, 1), (0, 16), (15, 33), (32, 64), (33, 130), (T - 1, T)):
        assert err(c.prefill(X, lo, hi, 0), want[lo:hi]) < 3e-5, (lo, hi)
    # rows of a tile that do not exist and positions not yet written (not-a-number values, large keys) leave no trace; scores far apart
    c = Case(scmx, T, H, G, d, dv, F32)
    c.q.mul_(12.0)
    c.fill()
    assert err(c.prefill(X, 40, 100, 0), c.want(list(range(40, 100)))) < 2e-4


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("M,N,K,tile,splits", [(24, 40, 128, 0, None), (23, 40, 24, 0, None), (130, 72, 132, 64, 1), (200, 300, 264, 128, 2), (300, 520, 257, 256, 1), (129, 256, 192, 256, 1),
                                               (513, 1000, 1100, 256, 5), (77, 33, 129, 0, None), (300, 160, 4096, 0, None), (128, 64, 2049, 64, 9), (40, 100, 1024, 0, None)])
def test_float32_product(X, M, N, K, tile, splits):      # noqa: F811
    """Sums of 64 values on tensor cores, float32 above: within 6e-7 of 64-bit sums in the 2-norm (measured 2.6e-7; plain
    float32 sums reach 5e-7 to 1.4e-6), whatever the tile, the ranges of K and the pitch of the rows."""
    g = torch.Generator("cuda").manual_seed(M * N + K)
    x, w = torch.randn(M, K + 3, generator=g, device="cuda")[:, :K], torch.randn(N, K, generator=g, device="cuda") * K ** -0.5
    lin = X.Linear(w)
    for rows in (x, x.contiguous()):
        y = lin(rows, tile=tile, splits=splits)
        assert y.shape == (M, N) and y.dtype == F32
        assert rel(y, rows.double() @ w.double().T) < 6e-7
    if N >= 40:
        assert torch.equal(lin.rows(8, 40)(x), X.Linear(w[8:40])(x))


def test_float32_product_activations(X):      # noqa: F811
    x, w = torch.randn(150, 160, device="cuda"), torch.randn(192, 160, device="cuda") * 0.1
    z = x.double() @ w.double().T
    act = X.XIELU(torch.tensor([0.3, -0.2]))
    want = torch.where(z > 0, act.a_pos * z * z, act.a_neg * (torch.expm1(z.clamp(max=0)) - z.clamp(max=0))) + 0.5 * z
    assert rel(X.Linear(w)(x, act=act), want) < 2e-6
    gate, up = z[:, :96], z[:, 96:]
    want = torch.nn.functional.gelu(gate, approximate="tanh") * up
    assert rel(X.Linear(X.GatedGELU.weight(w[:96], w[96:]))(x, act=X.GatedGELU()), want) < 2e-6


def test_float32_product_extreme_values(X):      # noqa: F811
    """Infinities and not-a-number values come out where float32 multiply-adds put them; the largest and smallest values keep their precision."""
    x, w = torch.randn(140, 300, device="cuda"), torch.randn(200, 300, device="cuda")
    x[3, 7], x[5, 1], x[9, 0], w[11, 20] = float("inf"), float("nan"), 3.4e38, float("-inf")
    x[9, 1:], w[:, 0] = 0.0, w[:, 0].clamp(-0.9, 0.9)
    x[20] *= 1e-30
    x[21] *= 1e34
    want = x.double() @ w.double().T
    for tile, splits in ((64, 1), (128, 2), (256, 1)):
        y = X.Linear(w)(x, tile=tile, splits=splits)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[y.isinf()].double(), want[want.isinf()])
        for r in (9, 20, 21, 30):
            ok = want[r].isfinite()
            assert rel(y[r][ok] / y[r][ok].abs().max(), want[r][ok] / y[r][ok].abs().max().double()) < 1e-6


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 8), (1, 1, 65, 9), (2, 2, 128, 128), (1, 1, 129, 7), (2, 1, 256, 24), (1, 1, 1, 1)])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dt", [BF, F32])
def test_delta_row_groups(X, H, G, d, dv, channel, dt):      # noqa: F811
    for cuts in ([50], [16, 17, 1, 15, 1], [33, 17]):
        c = DeltaCase(X, 50, H, G, d, dv, channel, dt)
        o, S = c.oracle()
        assert err(c.run(cuts, 1), o) < 2e-5 and err(c.state, S) < 2e-5, cuts
