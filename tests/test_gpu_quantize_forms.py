"""The quantizer's float32 screening against the oracle where it can go wrong: row lengths around a pass, ties and near-ties of the
candidates, values on the grid, the ends of the exponent range, values that are not finite, rows off the 16-byte boundary."""
import numpy as np
import pytest
import torch

from helpers import cuda

pytestmark = pytest.mark.gpu


def _check(scmx, oracle, wt):
    got = scmx.sc_format.quantize_device(wt)
    r = oracle.quantize(wt.double().cpu().numpy())
    for g, o in zip(got[:4], r):
        g = g.cpu().numpy()
        assert np.array_equal(g.view(np.uint32) if g.dtype == np.int32 else g, o)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [128, 384, 2048, 8064, 8192, 8320, 16640])
def test_row_lengths(scmx, oracle, dtype, k):
    rng = np.random.default_rng(k)
    w = rng.standard_normal((3, k)) * np.exp(rng.standard_normal((3, k)))
    w[1, 64:96] = 0
    w[2] = 0
    _check(scmx, oracle, cuda(w.astype(np.float32)).to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("exp", [-145, -128, -120, -60, 0, 60, 118, 122])
def test_grid_values_ties_and_exponents(scmx, oracle, dtype, exp):
    """Eighths up to 8: values on the grids of several candidates and in the middle between grid points, whose errors tie."""
    rng = np.random.default_rng(3)
    w = np.ldexp(rng.integers(-64, 65, (16, 512)) / 8.0, exp).astype(np.float32)
    w[1] = np.ldexp(rng.choice([0, 0.5, 1, 1.5, 2, 3, 4, 6], 512), exp).astype(np.float32)
    w[2, ::2] = np.nextafter(w[2, ::2], np.float32(0))
    w[3] *= np.ldexp(1.0, -20)
    w = w[np.isfinite(w).all(1)]
    _check(scmx, oracle, cuda(w).to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_not_finite_and_unaligned_as_the_float64_form(scmx, dtype):
    """NaN and infinities give what the float64 form gives (float64 input takes it), as do rows off the 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(1)
    w = (torch.randn((6, 1024), generator=g, device="cuda")).to(dtype)
    w[0, 5], w[1, 700], w[2, 40], w[3, :32] = float("nan"), float("inf"), float("-inf"), float("nan")
    off = torch.empty(w.numel() + 1, dtype=dtype, device="cuda")[1:].view(6, 1024).copy_(w)
    want = scmx.sc_format.quantize_device(w.double())
    for x in (w, off):
        for a, b in zip(scmx.sc_format.quantize_device(x), want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
