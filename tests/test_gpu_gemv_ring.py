"""GPU: the decode product (gemv_x_kernel) at the edges of its ring: rows shorter than a piece, a chunk and a slot, one row and odd numbers of them, rows
shared by several warps, rows so long that few warps stream, every epilogue, against float64.

Bound: every output is a float32 sum of K products of a bfloat16 or float32 weight and a float32 input in 32 lanes and two halves (K / 64 terms one after
another, then 6 levels), so its error is at most (K / 64 + 8) 2^-24 of the sum of the products' magnitudes; the epilogues below have slope at most 2."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8), (7, 8), (2, 1000), (33, 512), (301, 520), (160, 4096), (5, 6144), (4096, 128), (2500, 1024), (64, 51200), (99, 47104)]


def _case(N, K, dt, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + N * 7 + K)
    kp = (K + 7) // 8 * 8
    w = torch.zeros(N, kp, device="cuda", dtype=dt)
    w[:, :K] = torch.randn(N, K, generator=g, device="cuda").to(dt)
    return w, torch.randn(K, generator=g, device="cuda"), g


def _bound(w, x):
    K = x.numel()
    return (K / 64 + 8) * 2.0 ** -24 * (w[:, :K].double().abs() @ x.double().abs())


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,K", SHAPES)
def test_product(scmx, N, K, dt):
    L = scmx._lib
    w, x, _ = _case(N, K, dt)
    out = torch.full((N,), float("nan"), device="cuda")
    L.mcall("scmx_gemv_x", L.ptr(w), w.shape[1], int(dt == torch.float32), L.ptr(x), N, K, 0, 0.0, 0.0, None, None, None, 0, 0, L.ptr(out), L.stream())
    ref = w[:, :K].double() @ x.double()
    assert bool(((out.double() - ref).abs() <= _bound(w, x)).all())


@pytest.mark.parametrize("taps", [1, 2, 4, 5])
@pytest.mark.parametrize("N,C,K", [(1, 1, 64), (333, 200, 1024), (1200, 1200, 136), (9001, 9000, 64)])
def test_convolution_epilogue(scmx, N, C, K, taps):
    """taps up to 4 are kept in registers, more are read; the carried inputs move on by one."""
    L = scmx._lib
    w, x, g = _case(N, K, torch.bfloat16, 1)
    x = x * K ** -0.5
    cw, cb, tail = torch.randn(C, taps, generator=g, device="cuda"), torch.randn(C, generator=g, device="cuda"), torch.randn(C, taps - 1, generator=g, device="cuda")
    old, out = tail.clone(), torch.empty(N, device="cuda")
    L.mcall("scmx_gemv_x", L.ptr(w), w.shape[1], 0, L.ptr(x), N, K, 2, 0.0, 0.0, L.ptr(cw), L.ptr(cb), L.ptr(tail) if taps > 1 else None, C, taps, L.ptr(out), L.stream())
    y = w[:, :K].double() @ x.double()
    seq = torch.cat([old.double(), y[:C, None]], 1)
    c = (seq * cw.double()).sum(1) + cb.double()
    want = torch.cat([c * torch.sigmoid(c), y[C:]])
    # 2^-21: silu by the fast exponential and division, a few units in the last place
    size = torch.cat([(seq * cw.double()).abs().sum(1) + cb.double().abs(), torch.zeros(N - C, device="cuda", dtype=torch.float64)])
    bound = _bound(w, x) * torch.cat([2 * cw[:, -1].double().abs(), torch.ones(N - C, device="cuda", dtype=torch.float64)]) + 2.0 ** -20 * (size + want.abs())
    assert bool(((out.double() - want).abs() <= bound).all())
    assert torch.equal(tail[:, :taps - 2] if taps > 1 else tail, old[:, 1:] if taps > 1 else old)
    if taps > 1:
        assert bool(((tail[:, -1].double() - y[:C]).abs() <= _bound(w, x)[:C]).all())


@pytest.mark.parametrize("N,K", [(32, 8), (96, 1000), (6144, 1024), (12288, 512)])
def test_gate_up_epilogue(scmx, N, K):
    L = scmx._lib
    w, x, _ = _case(N, K, torch.bfloat16, 2)
    x = x * K ** -0.5
    out = torch.empty(N // 2, device="cuda")
    L.mcall("scmx_gemv_x", L.ptr(w), w.shape[1], 0, L.ptr(x), N, K, 3, 0.0, 0.0, None, None, None, 0, 0, L.ptr(out), L.stream())
    y = (w[:, :K].double() @ x.double()).view(-1, 2, 16)
    gate, up = y[:, 0].reshape(-1), y[:, 1].reshape(-1)
    want = torch.nn.functional.gelu(gate, approximate="tanh") * up
    b = _bound(w, x).view(-1, 2, 16)
    bound = 2 * b[:, 0].reshape(-1) * up.abs() + b[:, 1].reshape(-1) * (gate.abs() + 1) + 2.0 ** -19 * (gate.abs() + 1) * (up.abs() + 1)
    assert bool(((out.double() - want).abs() <= bound).all())
