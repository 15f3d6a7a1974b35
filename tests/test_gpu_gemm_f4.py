"""GPU: the products on digit planes (gemm_f4_kernel: tcgen05 kind::mxf4) against the oracle's and the packed-weight GEMM's bits: edges of token tiles, of weight tiles of
256 rows and of stages of 256 values, experts without rows, extreme codes (all of one sign, and the largest sums the accumulators hold), every epilogue; and the digits
themselves."""
import numpy as np
import pytest
import torch

from helpers import cuda

pytestmark = pytest.mark.gpu


def _weights(E, N, K, seed, extreme=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randint(-2 ** 31, 2 ** 31 - 1, (E, N * K // 8), generator=g, device="cuda").to(torch.int32)
    b = torch.randint(0, 256, (E, N, K // 128), generator=g, device="cuda").to(torch.uint8)
    if extreme:
        c.fill_(0x77777777), b.fill_(255)
    return c, b, torch.rand(E, N, generator=g, device="cuda") * 1e-3 + 1e-5, g


def _planes(dig, K):
    """int64 values of digit planes [3, rows, K / 8]."""
    nib = (dig.long()[..., None] >> torch.arange(0, 32, 4, device="cuda")) & 15
    return ((nib & 7) * (1 - 2 * (nib >> 3))).view(3, dig.shape[1], K)


def test_digits_of_every_code(scmx):
    M_ = scmx.sc_moe
    x = torch.arange(-128, 128, device="cuda").to(torch.int8).repeat(2, 1)
    d = _planes(M_.gather_digits(x, None, None, 2)[0], 256)
    assert int(d.abs().max()) <= 4
    assert torch.equal(d[0] + 8 * d[1] + 64 * d[2], x.long())


def test_factors(scmx):
    """Powers of two of the block codes in the tensor memory's order, several stacks in one launch, rows past N of a tile of 128 two."""
    M_ = scmx.sc_moe
    mats = [(1, 33, 128), (3, 256, 2048), (2, 300, 1152), (1, 128, 6144)]
    codes = [_weights(E, N, K, N)[1] for E, N, K in mats]
    for (E, N, K), b, f in zip(mats, codes, M_.f4_factors(*((b, *m) for b, m in zip(codes, mats)))):
        t, kb = -(-N // 128), K // 128
        got = f.view(E, t, kb, 32, 4, 4).permute(0, 1, 4, 3, 2, 5).reshape(E, t * 128, kb * 4)      # rows row % 32 + 32 (row / 32), blocks
        c = ((b.int()[..., None] >> torch.arange(0, 8, 2, device="cuda")) & 3).view(E, N, kb * 4)
        assert torch.equal(got[:, :N].int(), 128 + c) and bool((got[:, N:] == 128).all())


@pytest.mark.parametrize("M,K", [(1, 32), (33, 128), (40, 2048), (100, 1056), (7, 6144), (4097, 512), (300, 8192)])
def test_row_quantizer_digits(scmx, M, K):
    """Every form of the row quantizer (block, warps per row, segments): the digits of the INT8 rows that it writes otherwise, same scales."""
    S, L = scmx.sc_kernels, scmx._lib
    g = torch.Generator(device="cuda").manual_seed(K + M)
    x, w = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16), torch.randn(K, generator=g, device="cuda").to(torch.bfloat16)
    x[0] = 0
    for args, ref in (((), S.act_quant(x, M)), ((w, 1e-6), S.rmsnorm_quant(x, w, 1e-6, M))):
        dig, xs = S.quant_digits(x, *args)
        d = _planes(dig, K)
        assert torch.equal(d[0] + 8 * d[1] + 64 * d[2], ref[0].long()) and torch.equal(xs, ref[1])
    if K % 64 == 0:
        dig, xs = S.quant_digits(x.view(M, 2, K // 2).transpose(0, 1).contiguous(), segments=True)
        d = _planes(dig, K)
        assert torch.equal(d[0] + 8 * d[1] + 64 * d[2], S.act_quant(x, M)[0].long())


@pytest.mark.parametrize("extreme", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 32, 128), (16, 256, 256), (17, 288, 384), (80, 512, 640), (81, 256, 1024), (161, 64, 2048), (640, 4096, 256), (33, 96, 10240)])
def test_dense_bits(scmx, M, N, K, extreme):
    """INT32 totals against 64-bit sums, the other epilogues against the packed-weight GEMM.  `extreme`: every product 127 * 96 of one sign, the largest totals."""
    S, L, F, M_ = scmx.sc_kernels, scmx._lib, scmx.sc_format, scmx.sc_moe
    c, b, ws, g = _weights(1, N, K, M + N + K, extreme)
    xq = torch.randint(-127, 128, (M, K), generator=g, device="cuda").to(torch.int8)
    if extreme:
        xq.fill_(127)
        xq[-1] = -128
    xs, res = torch.rand(M, generator=g, device="cuda") * 0.01, torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16)
    dig, fac = M_.gather_digits(xq, None, None, M)[0], M_.f4_factors((b, 1, N, K))[0]
    wq = S.unpack_i8(c.view(-1), b.view(N, -1), N, K)
    tot = S.mm_f4(dig, c, fac, None, ws.view(-1), 0)
    assert torch.equal(tot.long(), (xq.double() @ wq.double().T).long())
    pad = -(-M // 128) * 128
    xqp, xsp, resp = torch.zeros(pad, K, dtype=torch.int8, device="cuda"), torch.zeros(pad, device="cuda"), torch.zeros(pad, N, dtype=torch.bfloat16, device="cuda")
    xqp[:M], xsp[:M], resp[:M] = xq, xs, res
    for epi in (1, 2, 3):
        if epi == 3 and N % 64:
            continue
        want = S.mm_epi(xqp, wq, xsp, ws.view(-1), epi, res=resp if epi == 2 else None)[:M]
        assert torch.equal(S.mm_f4(dig, c, fac, xs, ws.view(-1), epi, res), want), epi
    L.check_status()


def _bits(x):
    return x.contiguous().view(torch.int16 if x.dtype == torch.bfloat16 else torch.int32)


def _compare(scmx, xq, c, b, ws, N, K, seed):
    """Every epilogue, bit for bit (signs of zeros too), against the INT8 product, and the totals against 64-bit sums."""
    S, M_ = scmx.sc_kernels, scmx.sc_moe
    M, g = xq.shape[0], torch.Generator(device="cuda").manual_seed(seed)
    dig, fac, wq = M_.gather_digits(xq, None, None, M)[0], M_.f4_factors((b, 1, N, K))[0], S.unpack_i8(c.view(-1), b.view(N, -1), N, K)
    want = (xq.double() @ wq.double().T).long()
    assert torch.equal(S.mm_f4(dig, c, fac, None, ws, 0).long(), want)
    xs, res = torch.rand(M, generator=g, device="cuda") * 0.01, torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16)
    pad = -(-M // 128) * 128 - M
    xqp, xsp, resp = (torch.nn.functional.pad(t, (0, 0) * (t.dim() - 1) + (0, pad)) for t in (xq, xs, res))
    for epi in (1, 2, 3):
        ref = S.mm_epi(xqp, wq, xsp, ws, epi, res=resp if epi == 2 else None)[:M]
        assert torch.equal(_bits(S.mm_f4(dig, c, fac, xs, ws, epi, res)), _bits(ref)), epi
    scmx._lib.check_status()
    return want


@pytest.mark.parametrize("M,N,K", [(37, 128, 1024), (160, 256, 6144), (33, 64, 10240)])
def test_low_bits_of_large_sums(scmx, M, N, K):
    """Digits of -4 and -3 in the two lower planes times positive weights of every magnitude and block factor: plane sums between 2^15 and 2^22 whose low bits take every value
    (a plane whose accumulator dropped one would show), and single rows of the values with the largest digits, -36 = (-4, -4, 0) and 92 = (-4, -4, 2), times 96."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    nib = torch.randint(0, 8, (N, K // 8, 8), generator=g, device="cuda")
    nib[: N // 2, :, ::3] = 7                                   # half of the rows are heavy
    c = (nib << torch.arange(0, 32, 4, device="cuda")).sum(-1).to(torch.int32)
    b = torch.randint(0, 256, (1, N, K // 128), generator=g, device="cuda").to(torch.uint8)
    b[:, : N // 2] |= 0xAA
    c[0], b[0, 0] = 0x77777777, 255                             # one row of 96
    x = torch.tensor([-36, -35, -28, -27], device="cuda", dtype=torch.int8)[torch.randint(0, 4, (M, K), generator=g, device="cuda")]
    x[0], x[1], x[2], x[3], x[4] = -36, 92, -4, -32, 0
    want = _compare(scmx, x, c, b, torch.rand(N, generator=g, device="cuda") * 1e-3 + 1e-5, N, K, M)
    d0, d1 = (x.long() + 36) % 8 - 4, (x.long() + 36) // 8 % 8 - 4
    wq = scmx.sc_kernels.unpack_i8(c.view(-1), b.view(N, -1), N, K).double()
    for d in (d0, d1):
        sums = (d.double() @ wq.T).long().abs()
        assert int(sums.max()) == 384 * K and len(torch.unique(sums[5:] % 64)) == 64 and float((sums > 1 << 15).double().mean()) > 0.6
    assert int(want.abs().max()) == 92 * 96 * K


@pytest.mark.parametrize("K,N", [(5120, 128), (6144, 64), (10240, 192)])
def test_totals_around_two_to_the_24th(scmx, K, N):
    """Sums of the two lower planes on both sides of 2^24, where the epilogues go over to integers (36 * 96 * 4854 < 2^24 < 36 * 96 * 4855), with third planes of 0 and 2, and 64
    columns of any sign and magnitude that move them by single units."""
    c, b, ws, g = _weights(1, N, K, K, True)
    c.view(N, K // 8)[:, -8:] = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, 8), generator=g, device="cuda").to(torch.int32)
    x = torch.zeros(40, K, dtype=torch.int8, device="cuda")
    for r in range(40):
        x[r, :4854 - 15 + 5 * (r % 8)] = -36 if r < 24 else 92
        x[r, -64:] = torch.randint(-3, 4, (64,), generator=g, device="cuda").to(torch.int8)
    _compare(scmx, x, c, b, ws.view(-1), N, K, K)
    wq, low = scmx.sc_kernels.unpack_i8(c.view(-1), b.view(N, -1), N, K).double(), x.long() - 64 * ((x.long() + 36) // 64)
    past = (low.double() @ wq.T).abs() - 2.0 ** 24
    assert float(past.max()) > 0 > float(past.min()) and float(past.abs().min()) < 4000 and float(past.abs().max()) < 1 << 18


def test_swiglu_of_every_gate(scmx):
    """The epilogue's SiLU against sc_swiglu for all bfloat16 gates (finite and infinite ones equal), and scales that are infinite, not numbers or denormal against the INT8 product."""
    S, M_ = scmx.sc_kernels, scmx.sc_moe
    gate = torch.arange(65536, device="cuda").to(torch.int32).to(torch.int16).view(torch.bfloat16)
    K, N = 128, 64
    c = torch.zeros(N, K // 8, dtype=torch.int32, device="cuda")
    c[:, 0] = 1      # weight one half of two: every total is the activation's one
    b, xq = torch.zeros(1, N, 1, dtype=torch.uint8, device="cuda"), torch.zeros(65536, K, dtype=torch.int8, device="cuda")
    xq[:, 0] = 1
    got = S.mm_f4(M_.gather_digits(xq, None, None, 65536)[0], c.view(-1), M_.f4_factors((b, 1, N, K))[0], gate.float().contiguous(), torch.ones(N, device="cuda"), 3)
    want = S.sc_swiglu(gate, gate)
    fin = torch.isfinite(gate.float())
    assert torch.equal(got[fin].view(torch.int16), want[fin].view(torch.int16)[:, None].expand(-1, N // 2))
    assert bool(torch.isnan(got[torch.isnan(gate)]).all())
    inf = torch.isinf(gate.float())
    assert torch.equal(got[inf].isnan(), want[inf].isnan()[:, None].expand(-1, N // 2))
    assert torch.equal(got[inf].nan_to_num(7.0), want[inf].nan_to_num(7.0)[:, None].expand(-1, N // 2))
    wq = S.unpack_i8(c.view(-1), b.view(N, 1), N, K)
    scales = torch.tensor([float("inf"), float("-inf"), 3e38, -3e38, 1e-40, float("nan"), 1.0, 0.0], device="cuda").repeat(16)
    for q in (1, 0, -1):
        x8 = torch.zeros(128, K, dtype=torch.int8, device="cuda")
        x8[:, 0] = q
        for epi in (1, 3):
            new = S.mm_f4(M_.gather_digits(x8, None, None, 128)[0], c.view(-1), M_.f4_factors((b, 1, N, K))[0], scales, torch.ones(N, device="cuda"), epi)
            old = S.mm_epi(x8, wq, scales, torch.ones(N, device="cuda"), epi)
            assert torch.equal(new.isnan(), old.isnan())
            assert torch.equal(_bits(new[~new.isnan()]), _bits(old[~old.isnan()])), (q, epi)


@pytest.mark.parametrize("N,K", [(256, 256), (320, 1024), (2048, 128)])
@pytest.mark.parametrize("counts", [[0, 1, 0, 80, 81, 0], [5], [0, 0, 300], [16, 17, 160, 161, 33, 7, 250, 1, 0, 95]])
def test_grouped_bits(scmx, counts, N, K):
    M_, S = scmx.sc_moe, scmx.sc_kernels
    E, R = len(counts), sum(counts)
    c, b, ws, g = _weights(E, N, K, R + N)
    off = cuda(np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
    xq = torch.randint(-127, 128, (R, K), generator=g, device="cuda").to(torch.int8)
    xs = torch.rand(R, generator=g, device="cuda") * 0.01
    dig, fac = M_.gather_digits(xq, xs, None, R)[0], M_.f4_factors((b, E, N, K))[0]
    wq = M_.unpack_experts(c, b, N, K).view(E, N, K)
    starts = off.tolist()
    tot = M_.moe_mm_f4(dig, R, c, fac, ws, off, N, 0)
    for e in range(E):
        lo, hi = starts[e], starts[e + 1]
        assert torch.equal(tot[lo:hi].long(), (xq[lo:hi].double() @ wq[e].double().T).long())
    xp = torch.zeros(R + M_.TM, K, dtype=torch.int8, device="cuda")
    xp[:R] = xq
    tiles = [0]
    for n in counts:
        tiles.append(tiles[-1] + -(-n // M_.TM))
    ts = cuda(np.array(tiles, np.int32))
    for epi in (1, 3):
        want = M_.moe_mm_i8(xp, R, wq.view(E * N, K), ws, off, ts, -(-R // M_.TM) + E, N, epi, xs)
        assert torch.equal(M_.moe_mm_f4(dig, R, c, fac, ws, off, N, epi, xs), want), epi
    scmx._lib.check_status()


@pytest.mark.parametrize("kind,tokens", [("dense", 1), ("dense", 31), ("dense", 129), ("moe", 1), ("moe", 33), ("moe", 200)])
def test_prompts_equal_both_ways(scmx, monkeypatch, kind, tokens):
    """Prompts on digit planes against the INT8 products, at an empty cache and behind held positions: hidden states and cache rows bit for bit; a replaced attention is called."""
    HM = scmx.host_model
    if kind == "dense":
        FU = scmx.fused_qwen3
        model = HM.CausalLM(HM.ModelArgs(512, 768, 2, 4, 2, 128, 1e-6, 1e6, 512, True)).init_random(seed=4, scale=0.05).cuda()
        f, cls, limits = FU.FusedQwen3(model, FU.pack_model(model, on_device=True)), FU.FusedQwen3, ("F4_TOKENS", "F4_TOKENS_SMALL")
    else:
        FU = scmx.fused_olmoe
        model = HM.CausalLM(HM.ModelArgs(512, 256, 2, 4, 4, 128, 1e-5, 1e4, 512, False, 8, 2, False, "olmoe")).init_random(seed=4, scale=0.05).cuda()
        f, cls, limits = FU.FusedOlmoe(model, FU.pack_olmoe(model)), FU.FusedOlmoe, ("F4_ROWS",)
    ids = torch.randint(0, 512, (1, tokens), generator=torch.Generator().manual_seed(tokens)).cuda()
    out = {}
    for on in (True, False):
        for n in limits:
            monkeypatch.setattr(cls, n, 1 << 20 if on else -1)
        assert f._f4(tokens) is on
        cache, calls = f.make_cache(2 * tokens + 8), []
        own = f.sdpa
        hs = [f.hidden(ids, cache)]
        f.sdpa = lambda *a: calls.append(1) or own(*a)
        hs.append(f.hidden(ids, cache))
        f.sdpa = own
        assert len(calls) == 2
        out[on] = hs + [x[:, :2 * tokens] for c in cache for x in (c.k, c.v)]
    assert all(torch.equal(a, b) for a, b in zip(out[True], out[False]))
    scmx._lib.check_status()
