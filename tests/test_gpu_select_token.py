"""GPU: the greedy choice of a token, its list and its counters, against torch's argmax: sizes around the vector and cluster widths, equal
logits, not-a-number values, both logit types and an unaligned row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 7, 31, 4096, 4097, 32000, 50257, 151936])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("off", [0, 1])
def test_select_token(scmx, V, dt, off):
    L = scmx._lib
    tok, pos, count = torch.zeros(1, dtype=torch.long).cuda(), torch.full((1,), 40, dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    chosen = torch.full((8,), -1, dtype=torch.long).cuda()
    g = torch.Generator("cuda").manual_seed(V)
    rows = [torch.randn(V + off, generator=g, device="cuda").to(dt)[off:] for _ in range(9)]
    rows[1].fill_(-0.0)
    rows[1][V // 2:] = 0.0                          # equal values
    rows[2][-1] = float("inf")
    rows[3][V // 3] = rows[3][V // 2] = float("nan")
    rows[4].fill_(float("-inf"))
    rows[5].neg_().abs_().neg_()
    rows[6][V // 2:] = rows[6].max()
    want = [int(r.argmax()) for r in rows]
    for i, r in enumerate(rows):
        call = L.call if i % 2 else L.mcall
        call("scmx_select_token", L.ptr(r), int(dt == torch.float32), V, L.ptr(tok), L.ptr(pos), L.ptr(count), L.ptr(chosen), 8, L.stream())
        assert int(tok) == want[i], i
    assert chosen.tolist() == want[:8] and int(pos) == 49 and int(count) == 9
