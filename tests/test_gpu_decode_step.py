"""GPU: the one-kernel decode step (decode_step_kernel: rows as packets, weights in rings) bit for bit against the chain of kernels: one, two and four query heads per
key/value head, the smallest and the largest widths, one layer and several, positions on both sides of a split's edge, a full cache, and steps that share the scratch."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(1024, 1024, 1, 8, 8), (1024, 3072, 3, 8, 2), (2048, 6144, 2, 16, 8), (2048, 1024, 2, 32, 16), (3072, 2048, 2, 8, 4), (6144, 6144, 1, 16, 4)]


@pytest.mark.parametrize("D,F,layers,hq,hk", CASES)
def test_step_equals_chain(scmx, D, F, layers, hq, hk):
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC = mod("host_model"), mod("fused_qwen3"), mod("decode")
    model = HM.CausalLM(HM.ModelArgs(D, F, layers, hq, hk, 128, 1e-6, 1e6, 512, True)).init_random(seed=D + F, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    chain, mk = DEC.DecodeQwen3(fused, persistent=False), DEC.DecodeQwen3(fused, persistent=True)
    assert mk.persistent
    g = torch.Generator(device="cuda").manual_seed(D)
    for held, capacity in ((0, 40), (31, 40), (32, 40), (33, 34), (700, 720), (39, 40)):
        pair = [fused.make_cache(capacity) for _ in range(2)]
        for c, d in zip(*pair):
            for to, other in ((c.k, d.k), (c.v, d.v)):
                to.copy_(torch.randn(to.shape, generator=g, device="cuda").to(to.dtype))
                other.copy_(to)
            c.offset = d.offset = held
        tok = torch.tensor([[held % 512]], device="cuda")
        for _ in range(min(2, capacity - held)):      # twice on one cache: the second step follows the first one's epochs
            a, b = chain.step(tok, pair[0]), mk.step(tok, pair[1])
            assert torch.equal(a, b), (held, capacity)
        mk.check_status()
        for c, d in zip(*pair):
            assert torch.equal(c.k, d.k) and torch.equal(c.v, d.v)


@pytest.mark.parametrize("layers", [256, 257, 600])
def test_many_layers(scmx, layers):
    """More layers than a launch's table holds: a launch for every 256, the residual row handed on; two layers' weights in turn, a cache for every layer."""
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC = mod("host_model"), mod("fused_qwen3"), mod("decode")
    model = HM.CausalLM(HM.ModelArgs(1024, 1024, 2, 8, 4, 128, 1e-6, 1e6, 512, True)).init_random(seed=9, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    fused.layers = (fused.layers * layers)[:layers]
    chain, mk = DEC.DecodeQwen3(fused, persistent=False), DEC.DecodeQwen3(fused, persistent=True)
    pair = [sum((fused.make_cache(16) for _ in range(-(-layers // 2))), [])[:layers] for _ in range(2)]
    g = torch.Generator(device="cuda").manual_seed(layers)
    for c, d in zip(*pair):
        for to, other in ((c.k, d.k), (c.v, d.v)):
            to.copy_(torch.randn(to.shape, generator=g, device="cuda").to(to.dtype))
            other.copy_(to)
        c.offset = d.offset = 9
    tok = torch.tensor([[11]], device="cuda")
    for _ in range(2):
        assert torch.equal(chain.step(tok, pair[0]), mk.step(tok, pair[1]))
    mk.check_status()
    assert all(torch.equal(c.k, d.k) and torch.equal(c.v, d.v) for c, d in zip(*pair))


def test_step_after_one_that_gave_up(scmx):
    """The abort word of a step that gave up and its epochs do not reach the next one."""
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC = mod("host_model"), mod("fused_qwen3"), mod("decode")
    model = HM.CausalLM(HM.ModelArgs(1024, 1024, 2, 8, 4, 128, 1e-6, 1e6, 512, True)).init_random(seed=3, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    chain, mk = DEC.DecodeQwen3(fused, persistent=False), DEC.DecodeQwen3(fused, persistent=True)
    c1, c2 = fused.make_cache(16), fused.make_cache(16)
    for x in c1 + c2:
        x.k.zero_(), x.v.zero_()
    tok = torch.tensor([[5]], device="cuda")
    assert torch.equal(chain.step(tok, c1), mk.step(tok, c2))
    head = mk._mk["scratch"][:8].view(torch.int32)
    before = int(head[0])
    head[1] = 1                                       # as a thread that ran out of time leaves it
    assert torch.equal(chain.step(tok, c1), mk.step(tok, c2))
    assert head.tolist() == [before + (1 << 16) + 3, 0]
    mk.check_status()


def test_entry_with_scratch_of_its_own(scmx):
    """scmx_decode_step_dense, which allocates its scratch, against scmx_decode_step: the residual row bit for bit, alone and from a captured graph; its other buffers are not touched."""
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC, L = mod("host_model"), mod("fused_qwen3"), mod("decode"), scmx._lib
    model = HM.CausalLM(HM.ModelArgs(1024, 2048, 2, 8, 4, 128, 1e-6, 1e6, 512, True)).init_random(seed=3, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    dec, cache = DEC.DecodeQwen3(fused), fused.make_cache(16)
    for x in cache:
        x.k.normal_(), x.v.normal_()
    mk, pos, nsplit = dec._persistent_state(cache), torch.tensor([7], dtype=torch.int32, device="cuda"), dec.attn.nsplit
    h0 = torch.randn(1024, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    a, b = h0.clone(), h0.clone()
    other = [torch.zeros(64, dtype=torch.int32, device="cuda") for _ in range(6)]
    head = lambda h: (L.ptr(mk["table"]), 2, 1024, 2048, 8, 4, 128, 1e-6, 128 ** -0.5, L.ptr(fused.inv_freq), L.ptr(fused.rope_cs), fused.rope_cs.shape[0], 16,      # noqa: E731
                      L.ptr(pos), L.ptr(h))
    y, act, o, partials, counters, barrier = (L.ptr(x) for x in other)
    dense = lambda: L.call("scmx_decode_step_dense", *head(b), y, act, o, partials, nsplit, counters, barrier, L.ptr(mk["status"]), L.stream())      # noqa: E731
    L.call("scmx_decode_step", *head(a), L.ptr(mk["scratch"]), nsplit, L.ptr(mk["status"]), L.stream())
    dense()
    assert torch.equal(a, b) and not torch.equal(a, h0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dense()
    for _ in range(2):
        b.copy_(h0)
        graph.replay()
        assert torch.equal(a, b)
    dec.check_status()
    assert not any(bool(x.any()) for x in other)


@pytest.mark.parametrize("layers,link", [(2, 1), (2, 5), (2, 8), (258, 1286)])
def test_trace_of_arrivals(scmx, layers, link):
    """Both forms of the diagnostic: cycle counts of CTA 0 alone, and every CTA's arrival at one link, which lie between the marks of the step before and after it."""
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC, L = mod("host_model"), mod("fused_qwen3"), mod("decode"), scmx._lib
    model = HM.CausalLM(HM.ModelArgs(1024, 1024, 2, 8, 4, 128, 1e-6, 1e6, 512, True)).init_random(seed=3, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    fused.layers = fused.layers * (layers // 2)
    mk, cache = DEC.DecodeQwen3(fused), sum((fused.make_cache(16) for _ in range(layers // 2)), [])
    tok, n, sms = torch.tensor([[5]], device="cuda"), 9 * layers, torch.cuda.get_device_properties(0).multi_processor_count
    buf, lib = torch.zeros(n + sms + 1, dtype=torch.int64, device="cuda"), L.lib()
    try:
        for wanted in (0, link):
            buf.zero_()
            L.call("scmx_set_decode_trace", L.ptr(buf), n | wanted << 16)
            mk.step(tok, cache)
            marks, arrivals = buf[:n].tolist(), buf[n:n + sms].tolist()
            assert all(a < b for a, b in zip(marks, marks[1:])) or layers > 256      # (another launch, another SM)
            assert all(marks) and buf[-1] == 0
            if wanted:
                assert min(arrivals) > 0 and max(arrivals) - min(arrivals) < 10_000_000
            else:
                assert not any(arrivals)
    finally:
        lib.scmx_set_decode_trace(None, 0)
    mk.check_status()
