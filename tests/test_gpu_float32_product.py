"""GPU: float32 products of portions where they differ from a plain product: weights that change after the layer was built, weights taken in bands,
errors that have a sign, rows at the ends of the number range, values that are not finite, calls
that torch's own product has to take."""
import pytest
import torch

from test_gpu_hybrid_kernels import F32, X  # noqa: F401

pytestmark = pytest.mark.gpu


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("M", [1, 2, 24, 130])
def test_weights_changed_in_place(X, M):      # noqa: F811
    """A layer on the caller's memory follows it, in a captured graph too, and keeps nothing beside it."""
    x, w = torch.randn(M, 1024, device="cuda"), torch.randn(320, 1024, device="cuda") * 0.03
    held = torch.cuda.memory_allocated()
    lin = X.Linear(w)
    assert torch.cuda.memory_allocated() == held
    lin(x)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            z = lin(x)
    torch.cuda.current_stream().wait_stream(s)
    w.mul_(-0.5).add_(0.01)
    graph.replay()
    want = X.Linear(w.clone())(x)
    assert rel(want, x.double() @ w.double().T) < 1e-6
    assert torch.equal(lin(x), want) and torch.equal(z, want) and torch.equal(lin.rows(32, 96)(x), X.Linear(w[32:96].clone())(x))


@pytest.mark.parametrize("tile,splits", [(0, None), (64, 3), (128, 1), (256, 1)])
def test_bands_of_weights(X, monkeypatch, tile, splits):      # noqa: F811
    M, N, K = 70, 600, 1100      # bands of 256, 256 and 88 rows
    monkeypatch.setattr(X, "_band", lambda n, k: min(n, 256))
    x, w = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda") * K ** -0.5
    assert rel(X.Linear(w)(x, tile=tile, splits=splits), x.double() @ w.double().T) < 6e-7
    if splits in (None, 1):
        w = w[:576]
        z = x.double() @ w.double().T
        want = torch.nn.functional.gelu(z[:, :288], approximate="tanh") * z[:, 288:]
        assert rel(X.Linear(X.GatedGELU.weight(w[:288], w[288:]))(x, act=X.GatedGELU(), tile=tile, splits=splits), want) < 2e-6


@pytest.mark.parametrize("K", [256, 2048, 6144])
@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("tile", [64, 128, 256])
def test_error_has_little_sign(X, K, positive, tile):      # noqa: F811
    """No further from 64-bit sums than the library's float32 product, and nearly without a mean error.  An accumulator takes four additions, at a quarter, a
    half, three quarters and the whole of its sum, each cut by half a unit (2^-24 to 2^-23) in the mean: at most 2.5 * 2^-24 = 1.5e-7 in all."""
    g = torch.Generator("cuda").manual_seed(K)
    make = torch.rand if positive else torch.randn
    x, w = make(300, K, generator=g, device="cuda"), make(512, K, generator=g, device="cuda")
    want = x.double() @ w.double().T
    y = X.Linear(w)(x, tile=tile, splits=1)
    with X._full_float32():
        assert rel(y, want) <= rel(x @ w.T, want)
    assert abs(float(((y.double() - want) * want).sum() / (want * want).sum())) < 1.5e-7


@pytest.mark.parametrize("tile,splits", [(64, 1), (128, 3), (256, 1)])
@pytest.mark.parametrize("K", [301, 1028])
def test_scale_of_rows(X, K, tile, splits):      # noqa: F811
    """Rows of any size, to the ends of the number range, keep the precision of ordinary ones; the smallest results are off by a unit of the subnormal grid."""
    g = torch.Generator("cuda").manual_seed(K)
    x, w = torch.randn(160, K, generator=g, device="cuda"), torch.randn(200, K, generator=g, device="cuda")
    x *= torch.logspace(-37.5, 37.5, 160, device="cuda")[:, None]
    w *= torch.logspace(-37.5, 37.5, 200, device="cuda")[torch.randperm(200, generator=g, device="cuda")][:, None]
    x[7], w[9] = x[7].sign() * 2.0 ** -141, 0.0      # subnormal numbers, zeros
    x[8, 1:] = 0.0
    want, y = x.double() @ w.double().T, X.Linear(w)(x, tile=tile, splits=splits)
    top = torch.finfo(F32).max
    scale = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] / K ** 0.5      # of a typical sum of the row and column
    far = ((y.double() - want).abs() - splits * 2.0 ** -149) / scale.clamp(min=1e-300)
    ok = (want.abs() < 0.5 * top) & (scale < 0.01 * top)      # ranges of K are summed, so parts of a sum near the end may pass it
    assert float(far[ok].max()) < 5e-6 and ok.float().mean() > 0.4
    over = y[want.abs() > 2 * top]
    assert (over.isinf() if splits == 1 else ~over.isfinite()).all() and (y[:, 9] == 0).all()


@pytest.mark.parametrize("tile,splits", [(64, 1), (128, 3), (256, 1)])
@pytest.mark.parametrize("K", [129, 6144])
def test_values_not_finite(X, K, tile, splits):      # noqa: F811
    """Every row with an infinity, a few with not-a-number values: the answers of multiply-adds, and in a bounded time.  32 outputs of a row are K / 16 steps of 128 reads of 16 bytes a
    lane from shared memory, 4 cycles each, by 8 warps: 2.2 us, and 2 us for the loads before them; four such groups a warp 6.5 ms for K = 6144."""
    M, N = 160, 300
    x, w = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda")
    x[:, 1], x[3, 100], x[40, 5], w[17, 60], w[290, 128] = float("inf"), float("nan"), float("-inf"), float("nan"), float("-inf")
    x[100, 2] = 0.0
    w[200, 1] = 0.0                                # infinity times zero
    want, lin = x.double() @ w.double().T, X.Linear(w)
    y = lin(x, tile=tile, splits=splits)
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[~want.isnan()].double(), want[~want.isnan()])
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for bound, value in ((8.0, float("inf")), (1.0, float("nan"))):
        x[:] = value
        lin(x, tile=tile, splits=splits)
        a.record()
        lin(x, tile=tile, splits=splits)
        b.record()
        b.synchronize()
        assert a.elapsed_time(b) < bound


@pytest.mark.parametrize("M", [1, 2, 130])
def test_forms_that_only_torch_takes(X, M):      # noqa: F811
    """Columns first, rows that share memory, gradients, vmap, forward mode and autocast: the library's product, as before there was another."""
    K, N = 1024, 96
    w = torch.randn(N, K, device="cuda") * K ** -0.5
    lin, tol = X.Linear(w), 2e-6
    x = torch.randn(M, K, device="cuda")
    want = x.double() @ w.double().T
    assert rel(lin(x.T.contiguous().T), want) < tol
    assert rel(lin(x[:1].expand(M, K)), want[:1].expand(M, N)) < tol
    assert rel(torch.vmap(lambda r: lin(r[None])[0])(x), want) < tol
    primal, tangent = torch.func.jvp(lambda t: lin(t), (x,), (x * 2,))
    assert rel(primal, want) < tol and rel(tangent, 2 * want) < tol
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert lin(x).dtype == (x @ w.T).dtype
    x.requires_grad_()
    lin(x).sum().backward()
    assert rel(x.grad, w.double().sum(0).expand(M, K)) < tol
    with torch.no_grad():
        assert rel(lin(x), want) < tol
