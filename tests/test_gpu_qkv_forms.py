"""The q/k/v kernel's register form against the oracle: head sizes, head counts around what a CTA takes at once, one row and several,
with and without rotation, positions past the table, and the form through shared memory for unaligned rows."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [32, 64, 128, 256])
@pytest.mark.parametrize("hq,hk,full", [(1, 1, False), (3, 1, False), (16, 8, False), (5, 3, True), (11, 11, True), (16, 16, True), (16, 17, True)])
@pytest.mark.parametrize("mode", ["plain", "table", "past", "acc", "off"])
def test_forms_match_oracle(scmx, oracle, d, hq, hk, full, mode):
    S = scmx.sc_kernels
    L, ntot, eps, pos = (1 if mode == "past" else 3), (hq + 2 * hk) * d, 1e-6, 9
    if ntot * 4 + (hq + hk) * 4 + d * 4 > 48 * 1024:
        pytest.skip("a row that the kernels refuse")
    rng = np.random.default_rng(d + hq)
    qn = oracle.bf16_round(1 + 0.2 * rng.standard_normal(hq * d if full else d).astype(np.float32))
    kn = oracle.bf16_round(1 + 0.2 * rng.standard_normal(hk * d if full else d).astype(np.float32))
    inv = None if mode == "plain" else oracle.rope_inv_freq(d, 1e4)
    rope = None
    if inv is not None:
        rows = {"table": 64, "past": 4}.get(mode, 0)
        rope = (H.cuda(inv), pos) + ((S.rope_table(H.cuda(inv), rows),) if rows else ())
    if mode == "acc":
        acc = rng.integers(-200000, 200000, (L, ntot)).astype(np.int32)
        xs, ws = (rng.random(L).astype(np.float32) + 0.5) * 1e-3, (rng.random(ntot).astype(np.float32) + 0.5) * 1e-2
        want = oracle.qkv_epilogue_headnorm(acc, xs, ws, qn, kn, eps, L, hq, hk, d, full=full, inv_freq=inv, pos0=pos)
        src, xs, ws = H.cuda(acc), H.cuda(xs), H.cuda(ws)
    else:
        y = oracle.bf16_round(rng.standard_normal((L, ntot)).astype(np.float32) * 3)
        want = oracle.qkv_norm(y, qn, kn, eps, L, hq, hk, d, full=full, inv_freq=inv, pos0=pos)
        src, xs, ws = H.to_bf16_cuda(y), None, None
        if mode == "off":      # rows on a 4-byte boundary only
            src = torch.empty(src.numel() + 2, dtype=src.dtype, device="cuda")[2:].view(L, ntot).copy_(src)
    got = S._qkv_norm(src, xs, ws, H.to_bf16_cuda(qn), H.to_bf16_cuda(kn), eps, L, hq, hk, d, full, rope, None)
    for g, r in zip(got, want):
        assert np.array_equal(H.bf16_np(g), r)
