"""GPU: the sum of a token's expert rows with the norm that follows (moe_combine_norm_kernel) bit for bit against moe_combine and rmsnorm_quant_n one after the other: the
ends of a thread's vectors, one row and several, few and many experts a token, zero rows, and outputs that are left out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,topk", [(1, 8), (1, 1), (3, 9), (2, 32)])
@pytest.mark.parametrize("K", [8, 1032, 2048, 2056, 4128, 8192])
def test_bits(scmx, K, M, topk):
    M_, S = scmx.sc_moe, scmx.sc_kernels
    g = torch.Generator(device="cuda").manual_seed(K + 64 * M + topk)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)      # noqa: E731
    y, res, w, scores = rnd(M * topk, K), rnd(M, K), rnd(K), rnd(M, topk).abs()
    if M > 1:
        y[:topk], res[0] = 0, 0
    pos = torch.randperm(M * topk, generator=g, device="cuda").to(torch.int32)
    if M > 1:
        pos = torch.arange(M * topk, dtype=torch.int32, device="cuda")
    want = M_.moe_combine(y, pos, scores, res, w, 1e-5, M, quant=False)[0]
    xq, xs, xn = S.rmsnorm_quant_n(want, w, 1e-5, M)
    got = M_.combine_norm(y, pos, scores, res, w, 1e-5, normed=True)
    assert all(torch.equal(a, b) for a, b in zip(got, (want, xq, xs, xn)))
    h, q, s, n = M_.combine_norm(y, pos, scores, res, w, 1e-5, quant=False, normed=True)
    assert q is s is None and torch.equal(h, want) and torch.equal(n, xn)
    h, q, s, n = M_.combine_norm(y, pos, scores, res, w, 1e-5)
    assert n is None and torch.equal(q, xq) and torch.equal(s, xs)
    if K % 32 == 0:
        d, s = M_.combine_norm(y, pos, scores, res, w, 1e-5, quant="digits")[1:3]
        assert torch.equal(d, M_.gather_digits(xq, None, None, M)[0]) and torch.equal(s, xs)
