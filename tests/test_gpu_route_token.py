"""GPU: the router of one token in one kernel against the product, softmax and top-k done apart: experts around the warps of a cluster, widths around the
weights requested ahead, equal logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,D,k", [(1, 8, 1), (8, 256, 2), (63, 1024, 8), (64, 2048, 8), (65, 2056, 4), (130, 4096, 8), (257, 520, 3), (1024, 64, 16)])
def test_route_token(scmx, E, D, k):
    M_, g = scmx.sc_moe, torch.Generator("cuda").manual_seed(E + D)
    xn = torch.randn(1, D, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, D, generator=g, device="cuda") * 2 * D ** -0.5).to(torch.bfloat16)
    if E > 4:
        w[E // 2] = w[E - 1] = w[1]                  # equal logits: the lower expert first
    inds, scores = M_.route_token(xn, w, k)
    z = (xn.double() @ w.double().T).float()         # exact sums round to bfloat16 like float32 ones but for ties within 2^-16
    want_i, want_s = M_.router_topk(z.to(torch.bfloat16).float(), k)
    p = torch.softmax(z.to(torch.bfloat16).double(), 1)[0]
    step = float(z.abs().max()) * 2.0 ** -7         # one unit of a bfloat16 logit
    assert len(set(inds[0].tolist())) == k
    for i, s in zip(inds[0].tolist(), scores[0].tolist()):
        assert abs(s - float(p[i])) <= float(p[i]) * (step + 2.0 ** -8) + 1e-6
    kth = float(p.topk(k).values[-1])
    assert all(float(p[i]) >= kth * (1 - 2 * step) - 1e-9 for i in inds[0].tolist())
    if torch.equal(inds, want_i):
        assert (scores.float() - want_s.float()).abs().max() <= (step + 2.0 ** -7) * want_s.float().max()
    else:
        assert (inds != want_i).sum() <= 2


@pytest.mark.parametrize("E,D,k", [(1, 8, 1), (63, 1024, 8), (64, 2048, 8), (65, 2056, 4), (257, 520, 3), (1024, 8192, 16)])
def test_norm_route_token(scmx, E, D, k):
    """With the norm before it: the bits of rmsnorm_quant_n and route_token one after the other, a zero row included."""
    M_, S, g = scmx.sc_moe, scmx.sc_kernels, torch.Generator("cuda").manual_seed(E + D)
    x, nw, w = (torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16) for s in ((1, D), (D,), (E, D)))
    for row in (x, x * 1e-3, torch.zeros_like(x)):
        xq, xs, xn = S.rmsnorm_quant_n(row, nw, 1e-5, 1)
        want = (xq, xs, *M_.route_token(xn, w, k))
        assert all(torch.equal(a, b) for a, b in zip(M_.norm_route_token(row, nw, 1e-5, w, k), want))
