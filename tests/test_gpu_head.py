"""GPU: the output head of one row as a streaming product against 64-bit sums: rows around the CTAs' shares, widths around a set of loads, and where the
decoders must call the model's own head instead."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,K", [(1, 8), (7, 264), (591, 1024), (4737, 2048), (32000, 2056), (1200, 6400)])
def test_head(scmx, V, K):
    L, g = scmx._lib, torch.Generator("cuda").manual_seed(V + K)
    w, x = (torch.randn(V, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16), torch.randn(1, 1, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.empty(V, dtype=torch.bfloat16, device="cuda")
    L.call("scmx_head_bf16", L.ptr(w), K, L.ptr(x), V, K, L.ptr(out), L.stream())
    want = (w.double() @ x.double().view(-1))
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()      # one rounding to bfloat16


def test_own_heads_are_called(scmx):
    HM, head = scmx.host_model, scmx.sc_decode.head_product
    args = HM.ModelArgs(256, 512, 1, 2, 2, 128, 1e-6, 1e4, 500, True)
    with torch.device("cuda"):
        model = HM.CausalLM(args)
    h = torch.randn(1, 1, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        model.model.embed_tokens.weight.normal_()
        want = model.head(h)
        assert (head(model)(h).float() - want.float()).abs().max() <= 2.0 ** -6 * want.float().abs().max()
        assert torch.equal(head(model)(h.float()[..., :0].new_zeros(1, 1, 256).to(torch.bfloat16)), torch.zeros_like(want))

        class Own(HM.CausalLM):
            def head(self, h):
                return h[..., :3] * 2

        own = Own.__new__(Own)
        own.__dict__.update(model.__dict__)
        assert torch.equal(head(own)(h), h[..., :3] * 2)
        model.head = lambda h: h[..., :5]
        assert torch.equal(head(model)(h), h[..., :5])


def test_gradient_of_one_position(scmx):
    """Logits of one position carry a gradient where those of two do."""
    HM = scmx.host_model
    with torch.device("cuda"):
        model = HM.CausalLM(HM.ModelArgs(256, 512, 1, 2, 2, 128, 1e-6, 1e4, 500, False))
    model.lm_head.weight.requires_grad_()
    head = scmx.sc_decode.head_product(model)
    h = torch.randn(1, 1, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    head(h).float().sum().backward()
    assert torch.equal(model.lm_head.weight.grad[7], h.detach()[0, 0]) and h.grad is not None
    with torch.no_grad():
        assert (head(h).float() - model.head(h).float()).abs().max() <= 2.0 ** -6 * model.head(h).float().abs().max()


@pytest.mark.parametrize("N,K,dt", [(8, 8, torch.bfloat16), (32000, 1024, torch.bfloat16), (96, 6400, torch.bfloat16), (4096, 2048, torch.float32), (40, 100, torch.float32)])
def test_one_row(scmx, N, K, dt):
    """Products of one row run as streams of the weights, in both output types and from the last row of a portion."""
    X, g = scmx.sc_mixers, torch.Generator("cuda").manual_seed(N + K)
    w, x = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(dt), torch.randn(5, K, generator=g, device="cuda").to(dt)
    want = x[-1:].double() @ w.double().T
    lin = X.Linear(w)
    y = lin(x[-1:], torch.float32)
    assert y.dtype == torch.float32 and ((y.double() - want).norm() / want.norm()) < 2e-6
    if dt == torch.bfloat16:
        y = lin(x[-1:])
        assert y.dtype == dt and ((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
