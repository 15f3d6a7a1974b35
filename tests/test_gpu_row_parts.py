"""GPU: matrix-vector products that join their input row themselves against the row kernels followed by the product: widths around the two pieces per thread
and above (where the row kernels run), every form of the row and every epilogue."""
import pytest
import torch

from test_gpu_hybrid_kernels import BF, F32, X, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("K", [4, 36, 1024, 1028, 2044, 2048, 2052, 3000])
@pytest.mark.parametrize("form", ["norm", "add", "post", "average", "last", "final"])
@pytest.mark.parametrize("dt", [BF, F32])
def test_row_parts(X, K, form, dt):      # noqa: F811
    x, y, w, fw = rnd(1, 1, K), rnd(2, 1, K, scale=3.0), 1 + rnd(3, K, scale=0.2), 1 + rnd(4, K, scale=0.2)
    lin, N = X.Linear(rnd(5, 70, K, scale=K ** -0.5, dtype=dt)), 5
    xs, dwa = rnd(6, N + 1, 1, K), rnd(7, N, scale=0.4)
    avg, final, yy = {"norm": (None, None, None), "add": (None, None, y), "post": ((), None, y), "average": ((xs, dwa, True), None, y), "last": ((xs, dwa, False), None, y),
                      "final": ((xs, dwa, False), fw, y)}[form]
    out = torch.full_like(x, float("nan")) if yy is not None else None
    store = xs.clone()
    got = lin.vec(X.RowParts(x, yy, w, 0.7, 1e-3, out, avg, final))
    # the same in float64
    d = lambda t: t.double()      # noqa: E731
    rms = lambda t: t / torch.sqrt((t * t).mean() + 1e-3)      # noqa: E731
    if avg is None:
        r = d(x) + (0.7 * d(y) if yy is not None else 0)
        h = rms(r) * d(w)
    else:
        r = own = d(x) + d(w) * rms(d(y))
        if avg:
            r = (d(dwa)[:N - 1, None, None] * d(store)[:N - 1]).sum(0) + d(dwa)[N - 1] * r
            if avg[2]:
                assert rel(xs[N - 1], own) < 1e-6
                store[N - 1] = xs[N - 1]
        h = r if final is None else rms(r) * d(fw)
    assert torch.equal(xs, store)
    assert rel(got, (h @ d(lin.w[:, :K]).T).view(-1)) < 2e-6
    if out is not None:
        assert rel(out, r) < 1e-6


@pytest.mark.parametrize("K", [512, 2048])
def test_row_parts_epilogues(X, K):      # noqa: F811
    x, y, w = rnd(1, 1, K), rnd(2, 1, K), 1 + rnd(3, K, scale=0.2)
    part = lambda: X.RowParts(x, y, w, 0.5, 1e-4, torch.empty_like(x))      # noqa: E731
    row = part().joined()
    m = rnd(5, 320, K, scale=K ** -0.5, dtype=BF)
    for act, mat in ((X.XIELU(torch.tensor([0.3, -0.2])), m), (X.GatedGELU(), X.GatedGELU.weight(m[:160], m[160:]))):
        lin = X.Linear(mat)
        assert rel(lin.vec(part(), act=act), lin.vec(row, act=act)) < 2e-6
    cw, cb = rnd(9, 200, 4), rnd(10, 200)
    t1, t2 = rnd(11, 200, 3), rnd(11, 200, 3)
    lin = X.Linear(m)
    assert rel(lin.vec(part(), conv=(cw, cb, t1)), lin.vec(row, conv=(cw, cb, t2))) < 2e-6 and rel(t1, t2) < 2e-6
