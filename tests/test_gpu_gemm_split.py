"""GPU: INT8 products with K cut into ranges, bit for bit against the product in one piece: both kernels (CTA pairs, single CTAs), every epilogue, ranges of
unequal length, rows and columns off the tiles' edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,splits", [(128, 256, 1024, 2), (384, 2048, 2048, 4), (384, 544, 1040, 3), (256, 320, 6144, 8), (128, 64, 2176, 16), (640, 1024, 3072, 5),
                                          (128, 192, 256, 2)])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_split_product(scmx, M, N, K, splits, epi):
    if epi == 3 and N % 64:
        pytest.skip("pairs of gate and up columns")
    S, g = scmx.sc_kernels, torch.Generator("cuda").manual_seed(M + N + K)
    xq, wq = (torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((M, K), (N, K)))
    xs, ws = torch.rand(M, generator=g, device="cuda") * 1e-3, torch.rand(N, generator=g, device="cuda") * 1e-2
    res = torch.randn(M, N, generator=g, device="cuda").to(torch.bfloat16) if epi == 2 else None
    dt, n = (torch.int32, N) if epi == 0 else (torch.bfloat16, N // 2 if epi == 3 else N)
    one, cut = (torch.empty(M, n, dtype=dt, device="cuda") for _ in range(2))
    scales = (None, None) if epi == 0 else (xs, ws)
    S._mm_i8(xq, wq, M, N, K, epi, *scales, res, one, 1)
    S._mm_i8(xq, wq, M, N, K, epi, *scales, res, cut, splits)
    assert torch.equal(one, cut)
    if epi == 0:
        assert torch.equal(one.double(), xq.double() @ wq.double().T)
    scmx._lib.check_status()
