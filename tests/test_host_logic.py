"""CPU: host-side logic of the package (layout helpers, Format checks), the C-ABI library's exports, and the
argument validation every entry point performs before touching the GPU."""
import ctypes
import importlib.util
import os
import re

import numpy as np
import pytest
import torch
import torch.utils.flop_counter

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol(scmx):
    hdr = open(os.path.join(ROOT, "include", "scmx.h")).read()
    declared = set(re.findall(r"\b(scmx_[a-z0-9_]+)\s*\(", hdr))
    assert len(declared) >= 18
    h = ctypes.CDLL(scmx._lib.LIB_PATH)
    for name in declared:
        assert hasattr(h, name), f"{name} declared in include/scmx.h but not exported"
    assert declared == set(scmx._lib.SIGNATURES), "python binding and header disagree"
    assert scmx._lib.lib().scmx_abi_version() == 1


def test_pack_rows_decode_against_reference_vectors(scmx, golden):
    F = scmx.sc_format
    fmt = F.Format(block=16, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4)
    cc, bb, _ = F.pack_rows(golden["generic_code4"], golden["generic_bcode"], np.ones(8), fmt)
    assert np.array_equal(cc, golden["generic_codes"]) and np.array_equal(bb, golden["generic_bcodes"])
    assert np.array_equal(F.decode_numpy(cc, bb, 8, 256, fmt), golden["generic_q"])
    for tag in "abc":
        qw = golden[f"quantize_{tag}_qw"]
        assert np.array_equal(F.decode_numpy(golden[f"quantize_{tag}_codes"], golden[f"quantize_{tag}_bcodes"], *qw.shape), qw)


def test_from_shift_layout_roundtrip(scmx, golden):
    F = scmx.sc_format
    bc = golden["quantize_a_bcodes"]
    shifts = ((bc[..., None] >> (2 * np.arange(4, dtype=np.uint8))) & 3).reshape(bc.shape[0], -1)
    c, b, s = F.from_shift_layout(golden["quantize_a_codes"], shifts, golden["quantize_a_wscale"])
    assert np.array_equal(b, bc) and np.array_equal(c, golden["quantize_a_codes"])


def test_format_checks(scmx):
    F = scmx.sc_format
    assert F.DEFAULT.bits_per_weight(4096) == pytest.approx(4 + 2 / 32 + 32 / 4096)
    with pytest.raises(AssertionError):
        F.Format(block=12)
    with pytest.raises(AssertionError):
        F.Format(mult=(1, 2, 4, 8, 16))          # does not fit 2-bit block codes
    with pytest.raises(AssertionError):
        F.Format(mult=(1, 2, 4, 11))             # 12 * 11 > 127
    f = F.Format(block=16, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4).c_struct()
    assert (f.block, f.bc_bits, f.n_mult, f.mult[7]) == (16, 4, 8, 10)


def test_interleave_and_padding(scmx, golden):
    S = scmx.sc_kernels
    assert np.array_equal(S.interleave_gate_up(768), golden["perm_768"])
    assert [S.pad_rows(m) for m in (1, 128, 129, 200)] == [128, 128, 256, 256]


def test_entry_points_validate_before_launch(scmx):
    """Bad shapes and formats are rejected on the host with an error string; nothing reaches the GPU."""
    L = scmx._lib
    lib = L.lib()
    fmt = scmx.sc_format.DEFAULT.c_struct()
    bad = scmx.sc_format.DEFAULT.c_struct()
    bad.mult[3] = 11
    assert lib.scmx_act_quant(None, 4, 7, 4, None, None, None) == -1
    assert b"K % 8" in lib.scmx_last_error_string()
    assert lib.scmx_unpack_i8(None, None, 4, 256, bad, None, None) == -2
    assert b"INT8" in lib.scmx_last_error_string()
    assert lib.scmx_quantize_sc_mxfp4(None, 0, 4, 100, None, None, None, None, None, None) == -1
    assert lib.scmx_mm_i8(None, None, 128, 100, 256, 0, None, None, None, None, None, None) == -1
    assert lib.scmx_mm_i8(None, None, 128, 128, 256, 1, None, None, None, ctypes.c_void_p(16), ctypes.c_void_p(16), None) == -1
    assert lib.scmx_gemv(None, None, None, None, None, 6, 256, fmt, 1, None, None, 0, -1, 0, None, 0, None) == -1
    assert lib.scmx_route_sort(None, 4, 2, 2000, 128, None, None, None, None, None, None) == -5
    assert lib.scmx_moe_mm_i8(None, 10, None, None, ctypes.c_void_p(16), ctypes.c_void_p(16), 4, 128, 256, 0, None,
                              ctypes.c_void_p(16), 64, ctypes.c_void_p(16), None) == -1
    assert b"tm=64" in lib.scmx_last_error_string()
    assert lib.scmx_set_gemm_tile(64) == -1 and lib.scmx_set_gemm_tile(0) == 0
    with pytest.raises(L.ScmxError):
        L.call("scmx_act_quant", None, 4, 7, 4, None, None, None)


def test_no_cpu_fallback(scmx):
    import torch
    with pytest.raises(TypeError):
        scmx.sc_kernels.act_quant(torch.zeros(4, 64, dtype=torch.bfloat16))


def test_gemv_list_plan_geometry(scmx):
    """scmx_gemv_multi_plan is host code: tile shapes must respect the stage size (64 KB of codes, 2 KB of block codes), use at
    most 16 consumer warps, and number the tiles of the jobs consecutively.  Pointers only need to be non-NULL and aligned."""
    import ctypes
    L = scmx._lib
    shapes = [(4096, 2048), (2048, 2048), (12288, 2048), (2048, 6144), (100, 1024), (64, 8192), (1024, 3072), (4, 512)]
    jobs = (L.ScmxGemvJob * len(shapes))()
    for rec, (n, k) in zip(jobs, shapes):
        rec.codes = rec.bcodes = rec.wscale = rec.xq = rec.xscale = rec.out = 0x1000
        rec.N, rec.K, rec.epi = n, k, 1
    fmt = scmx.sc_format.DEFAULT.c_struct()
    assert L.lib().scmx_gemv_multi_plan(ctypes.byref(jobs), len(shapes), fmt) == 0, L.lib().scmx_last_error_string()
    tile0 = 0
    for rec, (n, k) in zip(jobs, shapes):
        tr, rg, sk, t0, nt, bcrow, kw = (rec.plan[i] for i in range(7))
        assert tr == 4 * rg and 1 <= rg * sk <= 16 and tr * k // 2 <= 65536 and tr * bcrow <= 2048
        assert kw * sk == k and kw % 32 == 0 and bcrow == k // 128
        assert t0 == tile0 and nt == -(-n // tr)
        tile0 += nt
    assert all(rec.plan[8] == tile0 for rec in jobs)
    assert jobs[0].plan[0] == 64 and jobs[3].plan[1] * jobs[3].plan[2] == 15      # K = 2048: 64-row tiles; K = 6144: 5 x 3 warps
    jobs[1].K = 128                                                                # one block-code byte per row: not a multiple of 4
    assert L.lib().scmx_gemv_multi_plan(ctypes.byref(jobs), len(shapes), fmt) == -5
    jobs[1].K = 100                                                                # not a multiple of 128
    assert L.lib().scmx_gemv_multi_plan(ctypes.byref(jobs), len(shapes), fmt) == -1
    jobs[1].K = 16384                                                              # beyond the activation slot of a stage
    assert L.lib().scmx_gemv_multi_plan(ctypes.byref(jobs), len(shapes), fmt) == -1


def test_packed_weight_gemm_format_rule(scmx):
    """scmx_w4_supported: the block codes of 128 weights must form one field of 8, 16 or 32 bits, K a multiple of 128."""
    F, L = scmx.sc_format, scmx._lib
    ok = lambda fmt, k: L.lib().scmx_w4_supported(fmt.c_struct(), k)   # noqa: E731
    assert ok(F.Format(), 2048) and ok(F.Format(block=16), 768) and ok(F.Format(block=16, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4), 2048)
    assert not ok(F.Format(), 2048 + 64)
    assert not ok(F.Format(block=64), 2048)            # 4 bits per 128 weights
    assert ok(F.Format(block=8), 2048)                 # 16 blocks x 2 bits = 32 bits
    assert not ok(F.Format(block=8, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4), 2048)      # 64 bits


def test_status_word_codes_have_texts(scmx):
    """Every code a kernel can leave in the status word has a description that names the waiting party (what check_status()
    raises with); unknown codes fall back to the number."""
    L = scmx._lib
    for code, word in ((1, "producer"), (2, "MMA"), (3, "MMA"), (4, "epilogue"), (6, "unpack"), (11, "GEMV"), (12, "GEMV"),
                       (20, "peer barrier")):
        assert word in L.describe_status(code), code
    assert L.describe_status(1000) == "decode step: layer 0 waiting for its input row"
    assert L.describe_status(1000 + 5 * 27 + 3) == "decode step: layer 27 waiting for its residual row after attention"
    assert L.describe_status(77) == "code 77" and L.describe_status(103) == "code 103"


def test_calls_that_torch_has_to_see(scmx):
    """A kernel takes the place of a torch operation only where nothing records, transforms or recasts it."""
    unseen, x, w = scmx._lib.unseen, torch.randn(3), torch.nn.Parameter(torch.randn(3))
    seen = []
    assert unseen(x, x) and not unseen(x, w)
    with torch.no_grad():
        assert unseen(x, w)
        torch.vmap(lambda t: seen.append(unseen(t)) or t)(x)
        torch.func.jvp(lambda t: seen.append(unseen(t)) or t, (x,), (x,))
        with torch.autograd.forward_ad.dual_level():
            seen.append(unseen(x))
        torch.set_autocast_enabled("cuda", True)      # as torch.autocast does where there is a GPU
        seen.append(unseen(x))
        torch.set_autocast_enabled("cuda", False)
        with torch.utils.flop_counter.FlopCounterMode(display=False):
            seen.append(unseen(x))
        torch.jit.trace(lambda t: seen.append(unseen(t)) or t, x, check_trace=False)

        class Own(torch.Tensor):
            pass

        seen.append(unseen(x.as_subclass(Own)))
    assert seen == [False] * 7


@pytest.mark.parametrize("tied", [False, True])
def test_heads_that_want_the_call(scmx, monkeypatch, tied):
    """The head's matrix is handed out only while `head` is a product with it and nobody watches or replaces the call."""
    HM = scmx.host_model
    model = HM.CausalLM(HM.ModelArgs(256, 512, 1, 2, 2, 128, 1e-6, 1e4, 500, tied))
    matrix = model.model.embed_tokens.weight if tied else model.lm_head.weight
    assert model.head_weight() is matrix
    with monkeypatch.context() as m:
        m.setattr(HM.CausalLM, "head", lambda self, h: h)
        assert model.head_weight() is None
    with monkeypatch.context() as m:
        m.setitem(model.__dict__, "head", lambda h: h)
        assert model.head_weight() is None
    if not tied:
        with monkeypatch.context() as m:
            m.setitem(model.lm_head.__dict__, "forward", lambda h: h)
            assert model.head_weight() is None
        with monkeypatch.context() as m:
            m.setattr(torch.nn.Linear, "forward", lambda self, h: h)
            assert model.head_weight() is None
        nn = torch.nn.modules.module
        for hook in (model.lm_head.register_forward_hook, model.lm_head.register_forward_pre_hook, nn.register_module_forward_hook, nn.register_module_forward_pre_hook,
                     model.lm_head.register_full_backward_hook, nn.register_module_full_backward_hook):
            handle = hook(lambda *a: None)
            assert model.head_weight() is None, hook
            handle.remove()
    assert model.head_weight() is matrix
    # and the product itself asks torch where a gradient, a transform or a mode would miss it
    h, seen = torch.zeros(1, 1, 256, dtype=torch.bfloat16), []
    monkeypatch.setitem(model.__dict__, "head", lambda t: seen.append(t.requires_grad) or t)
    monkeypatch.setattr(model, "head_weight", lambda: matrix)
    product = scmx.sc_decode.head_product(model)
    product(h)                                  # the weight may want a gradient
    with torch.no_grad():
        torch.vmap(product)(h[None])
    assert len(seen) == 2


def test_replaced_attention_is_called(scmx, monkeypatch):
    """A prompt's attention is read head by head only where it is this library's own function."""
    HM, S = scmx.host_model, scmx.sc_kernels
    monkeypatch.setattr(S, "act_quant", lambda x, rows: x)
    monkeypatch.setattr(S, "act_quant_seg", lambda x, rows: x.transpose(0, 1).reshape(x.shape[1], -1))
    q, answer = torch.randn(2, 3, 8), torch.randn(3, 16)
    assert torch.allclose(scmx.fused_qwen3.attend_quant(HM.sdpa, q, q, q, 1.0, 128), HM.sdpa(q, q, q, 1.0, True))
    own = lambda *a: answer      # noqa: E731
    assert scmx.fused_qwen3.attend_quant(own, q, q, q, 1.0, 128) is answer
    monkeypatch.setattr(HM, "sdpa", own)
    assert scmx.fused_qwen3.attend_quant(HM.sdpa, q, q, q, 1.0, 128) is answer


def test_plans_count_the_device(scmx, monkeypatch):
    """Tiles and ranges of K are planned for the current device's multiprocessors, also after another device has been asked about."""
    L, S, X = scmx._lib, scmx.sc_kernels, scmx.sc_mixers

    class Of:
        def __init__(self, dev):
            self.multi_processor_count = (148, 20)[dev]

    dev = [0]
    monkeypatch.setattr(L, "_sms", {})
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: dev[0])
    monkeypatch.setattr(torch.cuda, "get_device_properties", Of)
    plans = lambda: (S._ranges(256, 2048, 6144, L.sm_count()), X._plan(77, 1024, 3072, None, L.sm_count()), X._plan_f32(77, 1024, 3072, None, L.sm_count()))      # noqa: E731
    large = plans()
    assert large[0] == 4 and large[1][1] > 1 and large[2][1] > 1
    dev[0] = 1
    small = plans()
    assert small[0] == 1 and small[1] != large[1] and small[2] != large[2]
    dev[0] = 0
    assert plans() == large


def test_structures_are_defined_once(scmx):
    """The sources of one library share a namespace, so a structure of the same name in two of them would be two definitions of one class."""
    spec = importlib.util.spec_from_file_location("scmx_build", os.path.join(ROOT, "mxfp4-int8-m5_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    for which in build.LIBS:
        where = {}
        for path in set(build._deps(which)):
            for name in set(re.findall(r"^\s*(?:template <[^>]*>\s*)?struct (\w+)(?:<[^;{]*>)?\s*\{", open(path).read(), re.M)):
                assert where.setdefault(name, path) == path, (name, path, where[name])


def test_two_passes_on_request(scmx):
    """A mixture's prompts of few rows per expert run on packed weights unless two passes are asked for, by any true value."""
    fused = scmx.fused_olmoe.FusedOlmoe.__new__(scmx.fused_olmoe.FusedOlmoe)
    fused.args = scmx.host_model.ModelArgs(2048, 1024, 1, 16, 16, 128, num_experts=64, num_experts_per_tok=8)
    for two_pass, packed in (("auto", True), (False, True), (True, False), (1, False), (np.True_, False)):
        fused.two_pass = two_pass
        assert fused._packed(64 * 479) is packed and not fused._packed(64 * 480)


def test_replaced_router_is_called(scmx, monkeypatch):
    """A decode step asks a `route` that was replaced on the object, in a subclass or in the class, not the kernel for one token."""
    FO = scmx.fused_olmoe
    monkeypatch.setattr(scmx.sc_moe, "route_token", lambda xn, w, k: "kernel")

    class Own(FO.FusedOlmoe):
        def route(self, layer, xn, M):
            return "own"

    class Layer:
        class mlp:
            gate = torch.nn.Linear(64, 8, bias=False, dtype=torch.bfloat16)

    plain, own = (c.__new__(c) for c in (FO.FusedOlmoe, Own))
    plain.args = own.args = scmx.host_model.ModelArgs(64, 128, 1, 1, 1, 64, num_experts=8, num_experts_per_tok=2)
    xn = torch.zeros(1, 64, dtype=torch.bfloat16)
    assert plain.route_token(Layer, xn) == "kernel" and own.route_token(Layer, xn) == "own"
    plain.route = lambda layer, xn, M: "object"
    assert plain.route_token(Layer, xn) == "object"
    del plain.route
    monkeypatch.setattr(FO.FusedOlmoe, "route", lambda self, layer, xn, M: "class")
    assert plain.route_token(Layer, xn) == "class"


def test_replaced_router_of_a_token_is_called(scmx, monkeypatch):
    """Nor does a step's norm with the router pass by a `route` or `route_token` that was replaced."""
    FO, S, M_ = scmx.fused_olmoe, scmx.sc_kernels, scmx.sc_moe
    monkeypatch.setattr(M_, "norm_route_token", lambda *a: "kernel")
    monkeypatch.setattr(S, "rmsnorm_quant_n", lambda h, w, eps, M: ("q", "s", h))

    class Layer:
        post_attention_layernorm = torch.nn.LayerNorm(64)

        class mlp:
            gate = torch.nn.Linear(64, 8, bias=False, dtype=torch.bfloat16)

    class Own(FO.FusedOlmoe):
        def route_token(self, layer, xn):
            return "own", "scores"

    def make(cls=FO.FusedOlmoe):
        f = cls.__new__(cls)
        f.args, f.eps = scmx.host_model.ModelArgs(64, 128, 1, 1, 1, 64, num_experts=8, num_experts_per_tok=2), 1e-5
        return f

    h, plain = torch.zeros(1, 64, dtype=torch.bfloat16), make()
    assert plain.norm_route_token(Layer, h) == "kernel" and make(Own).norm_route_token(Layer, h) == ("q", "s", "own", "scores")
    plain.route = lambda layer, xn, M: ("route", M)
    assert plain.norm_route_token(Layer, h) == ("q", "s", "route", 1)
    del plain.route
    plain.route_token = lambda layer, xn: ("token", "scores")
    assert plain.norm_route_token(Layer, h) == ("q", "s", "token", "scores")
    del plain.route_token
    monkeypatch.setattr(FO.FusedOlmoe, "route_token", lambda self, layer, xn: ("class", "scores"))
    assert plain.norm_route_token(Layer, h) == ("q", "s", "class", "scores")


def test_replaced_quantizer_is_called(scmx, monkeypatch):
    """The attention output of a prompt goes to an `act_q` that was replaced on the object, in a subclass or in the class."""
    FQ = scmx.fused_qwen3
    monkeypatch.setattr(FQ, "attend_quant", lambda *a: ("kernel", "scales"))

    class Own(FQ.FusedQwen3):
        def act_q(self, x, Mp=None, nt=256, down=False):
            return "own", "scales"

    class At:
        scale = 1.0

    plain, own = (c.__new__(c) for c in (FQ.FusedQwen3, Own))
    for f in (plain, own):
        f.rot, f.record, f.record_layers, f.sdpa = False, None, (), lambda *a: "rows"
        f._qkv = lambda *a: (None, None, None)
    ask = lambda f: f._attention(0, At, None, None, None, None, 3, 128)[1]      # noqa: E731
    assert ask(plain) == "kernel" and ask(own) == "own"
    plain.act_q = lambda x, Mp: ("object", "scales")
    assert ask(plain) == "object"
    del plain.act_q
    monkeypatch.setattr(FQ.FusedQwen3, "act_q", lambda self, x, Mp: ("class", "scales"))
    assert ask(plain) == "class"


def test_shared_format_struct(scmx):
    """The struct handed to the kernels follows DEFAULT, is never the caller's own, and formats given as lists still work."""
    F, S = scmx.sc_format, scmx.sc_kernels
    old = F.DEFAULT
    try:
        for fmt in (F.Format(), F.Format(block=16, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4), F.Format(code_mag=[0, 1, 2, 3, 4, 6, 8, 12], mult=[1, 2, 4])):
            S.set_format(fmt)
            fmt.c_struct().block = 99
            assert bytes(F.c_default()) == bytes(fmt.c_struct())
    finally:
        S.set_format(old)


@pytest.mark.parametrize("layers", [1, 256, 257])
def test_decode_step_form(scmx, layers):
    """The one-kernel step takes any number of layers."""
    from types import SimpleNamespace as NS
    args = scmx.host_model.ModelArgs(1024, 1024, layers, 8, 4, 128, 1e-6, 1e6, 512, True)
    fused = NS(epilogue="gemm", model=NS(), args=args, inv_freq=torch.zeros(64), fmt=scmx.sc_format.Format())
    assert scmx.decode.DecodeQwen3(fused, head=lambda x: x).persistent


def test_decode_step_on_fewer_multiprocessors(scmx, monkeypatch):
    """A decoder on a partition of the device takes the chain of kernels where the one-kernel step would refuse its shares."""
    from types import SimpleNamespace as NS
    A, D = scmx.host_model.ModelArgs, scmx.decode.DecodeQwen3
    narrow, wide = A(1024, 1024, 1, 8, 4, 128, 1e-6, 1e6, 512, True), A(6144, 6144, 1, 32, 8, 128, 1e-6, 1e6, 512, True)
    fits = lambda a, nsplit: [n for n in (4, 8, 16, 31, 32, 63, 64, 148, 256, 257) if D._shares_fit(a, nsplit, n)]      # noqa: E731
    assert fits(narrow, 1) == [8, 16, 31, 32, 63, 64, 148, 256] and fits(narrow, 32) == [148, 256]
    assert fits(wide, 1) == [32, 63, 64, 148, 256, 257] and fits(wide, 18) == [148, 256, 257]
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    fused = NS(epilogue="gemm", model=NS(), args=narrow, inv_freq=torch.zeros(64), fmt=scmx.sc_format.Format())
    for sms, one_kernel in ((148, True), (64, False)):      # 4 heads of 32 splits
        monkeypatch.setattr(scmx._lib, "sm_count", lambda: sms)
        assert D(fused, head=lambda x: x).persistent is one_kernel


def test_prompts_on_digit_planes(scmx):
    """Which prompts of a dense decoder run on digit planes: few tokens, the default format, and none of the class's own steps replaced."""
    from types import SimpleNamespace as NS
    FQ, F, S = scmx.fused_qwen3, scmx.sc_format, scmx.sc_kernels

    class Own(FQ.FusedQwen3):
        def rms_q(self, h, nw, Mp=None):
            return "own", "scales"

    def make(cls=FQ.FusedQwen3, width=4096, K=2048, **kw):
        f = cls.__new__(cls)
        f.layers, f.epilogue, f.resident, f.rot, f.record = [(None, {g: NS(N=width, K=K) for g in FQ.GROUPS})], "gemm", False, False, None
        f.__dict__.update(kw)
        return f

    limit, small = FQ.FusedQwen3.F4_TOKENS, FQ.FusedQwen3.F4_TOKENS_SMALL
    assert [make(width=8192)._f4(n) for n in (0, 1, limit, limit + 1)] == [False, True, True, False]
    for width, most in ((5120, limit), (5119, 600), (4352, 600), (4351, 448), (4096, 448), (4095, small)):      # weights of a layer: 4 x width x 2048
        assert [make(width=width)._f4(n) for n in (most, most + 1)] == [True, False], width
    assert [make(width=1024)._f4(n) for n in (small, small + 1)] == [True, False]
    assert not any(make(**kw)._f4(16) for kw in (dict(cls=Own), dict(K=2048 + 64), dict(K=10240), dict(epilogue="row"), dict(resident=True), dict(rot="down"),
                                                 dict(record={}), dict(act_q=lambda x, Mp: None), dict(_rec=lambda *a: None)))
    old = F.DEFAULT
    try:
        S.set_format(F.Format(block=16, mult=(1, 2, 3, 4, 5, 6, 8, 10), bc_bits=4))
        assert not make()._f4(16)
    finally:
        S.set_format(old)


class _Clock:
    """Streams and events that know which operations they come after."""

    class Stream:
        cuda_stream = 0

        def __init__(self, **kw):
            self.before = set()

        def do(self, op):
            self.before.add(op)

        def wait_event(self, e):
            self.before |= e.before

        def wait_stream(self, other):
            self.before |= other.before

    class Event:
        before = frozenset()

        def record(self, stream):
            self.before = frozenset(stream.before)


@pytest.mark.parametrize("overlap,group,count", [(True, 1, 1), (True, 1, 5), (True, 2, 5), (False, 1, 3)])
def test_ring_on_another_stream(scmx, monkeypatch, overlap, group, count):
    """A pass on another stream decodes into the ring's buffers only after every product of the pass before that read them, and so on to and fro."""
    FD, S = scmx.fused_dense, scmx.sc_kernels
    current, capturing = [None], [False]
    for name, fake in dict(Stream=_Clock.Stream, Event=_Clock.Event, current_stream=lambda: current[0], is_current_stream_capturing=lambda: capturing[0]).items():
        monkeypatch.setattr(torch.cuda, name, fake)
    ring = FD.DecodeRing(64, "cpu", overlap, group)
    readers, turn = {}, [0]

    def unpack(codes, bc, N, K, out, stream):
        on = ring.side if overlap else current[0]
        if not capturing[0]:
            assert readers.get(out.data_ptr(), set()) <= on.before
        on.do(("decode", out.data_ptr(), turn[0]))

    monkeypatch.setattr(S, "unpack_i8", unpack)
    a, b, c = (_Clock.Stream() for _ in range(3))
    for stream, captured in ((a, False), (a, False), (b, False), (c, True), (c, False), (a, False), (b, False)):
        current[0], capturing[0] = stream, captured
        ring.begin([(None, None, None, 8, 8)] * count)
        for g in range(count):
            turn[0] += 1
            w = ring.weight(g).data_ptr()
            stream.do(("read", w, turn[0]))
            if not captured:
                readers.setdefault(w, set()).add(("read", w, turn[0]))
            ring.released(g)
        ring.end()


def test_generation_keeps_what_its_graph_names(scmx, monkeypatch):
    """Steps on other caches replace the one-kernel step's tables; those of a captured generation stay alive and are the decoder's again when it is replayed."""
    import contextlib
    import weakref
    from types import SimpleNamespace as NS

    class Stream:
        def wait_stream(self, other):
            pass

    class Graph:
        def replay(self):
            assert self.table() is not None, "replayed on a table that was freed"

    class Decoder(scmx.decode._Decoder):
        replayable = True

        def __init__(self):
            self._graph = self._mk = None

        def _step(self, tok, cache, pos):
            if self._mk is None or self._mk["cache"] is not cache:
                self._mk = dict(cache=cache, table=torch.zeros(4))
            Graph.table = weakref.ref(self._mk["table"])
            return torch.zeros(1, 1, 8)

        def _select(self, *a):
            pass

    nothing = lambda *a, **kw: contextlib.nullcontext()      # noqa: E731
    for name, fake in dict(Stream=lambda device: Stream(), current_stream=Stream, stream=nothing, synchronize=lambda: None, CUDAGraph=Graph, graph=nothing).items():
        monkeypatch.setattr(torch.cuda, name, fake)
    make = lambda: [NS(offset=3, capacity=16, carried=lambda: [])]      # noqa: E731
    a, b, dec, tok = make(), make(), Decoder(), torch.zeros(1, 1, dtype=torch.long)
    dec.generate(tok, a, 2)
    first = dec._mk
    table = Graph.table
    dec.step(tok, b)
    assert dec._mk is not first
    del first
    Graph.table = table
    dec.generate(tok, a, 2)
    assert dec._mk["table"] is table()
