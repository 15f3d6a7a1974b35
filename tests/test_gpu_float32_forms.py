"""GPU: the float32 forms of retention and differential attention at the edges of their tiles, against the float64 oracle: heads up to the
register limits and one above, portions around 16 tokens, 16 queries and 32 keys, value sizes of one and two column groups."""
import pytest
import torch

from test_gpu_hybrid_kernels import BF, F32, Case, X, err, ret_case, run_ret  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,dv,dims", [(2, 64, 16, 64), (1, 65, 17, 6), (2, 128, 256, 128), (1, 129, 15, 128), (2, 256, 40, 0), (1, 257, 33, 254)])
@pytest.mark.parametrize("dt", [BF, F32])
def test_retention_row_groups(X, H, d, dv, dims, dt):      # noqa: F811
    T = 50
    case = ret_case(X, T, H, d, dv, dims, dt)
    for cuts in ([T], [16, 17, 1, 15, 1], [31, 19]):
        o, S = run_ret(X, case, H, d, dv, dims, cuts, 1)
        assert err(o, case[1][0]) < 2e-5 and err(S, case[1][1]) < 2e-5


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 128), (2, 2, 4, 4), (3, 1, 36, 132), (2, 1, 128, 256), (1, 1, 12, 260), (4, 2, 66, 128)])
def test_differential_attention_tiles(X, scmx, H, G, d, dv):      # noqa: F811
    T = 150
    c = Case(scmx, T, H, G, d, dv, F32)
    c.fill()
    want = c.want(list(range(T)))
    for lo, hi in ((0, T), (0, 1), (0, 16), (15, 33), (32, 64), (33, 130), (T - 1, T)):
        assert err(c.prefill(X, lo, hi, 0), want[lo:hi]) < 3e-5, (lo, hi)
    # rows of a tile that do not exist and positions not yet written (not-a-number values, large keys) leave no trace; scores far apart
    c = Case(scmx, T, H, G, d, dv, F32)
    c.q.mul_(12.0)
    c.fill()
    assert err(c.prefill(X, 40, 100, 0), c.want(list(range(40, 100)))) < 2e-4
