"""GPU: bounded device-side waits that run out.  scmx_peer_barrier is called for a world of two ranks on two local flag
arrays that nobody else signals, with the wait limit lowered to 2 ms: the kernel must return by itself, leave code 20 in the
status word, and check_status() must raise.  A one-kernel decode step is given attention over so many positions by so few CTAs that the others run
out of a limit of 1 us meanwhile.  Nothing faults, traps or spins without a limit."""
import ctypes
import importlib
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_peer_barrier_wait_runs_out_and_reports(scmx):
    L = scmx._lib
    flags = [torch.zeros(8, dtype=torch.int32, device="cuda") for _ in range(2)]
    peers = (ctypes.c_void_p * 8)(flags[0].data_ptr(), flags[1].data_ptr(), *([None] * 6))
    epoch = torch.zeros(1, dtype=torch.int32, device="cuda")
    status = L.status_buffer()
    status.zero_()
    L.call("scmx_set_wait_limit_ns", 2_000_000)
    try:
        t0 = time.perf_counter()
        L.call("scmx_peer_barrier", peers, 0, 2, L.ptr(epoch), L.ptr(status), L.stream())
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    finally:
        L.call("scmx_set_wait_limit_ns", 2_000_000_000)
    assert dt < 1.0, f"the barrier took {dt:.3f} s with a 2 ms limit"
    assert status[0].item() == 20 and status[1].item() == 0      # code 20 = peer barrier, reported by rank 0
    assert epoch.item() == 1 and flags[1][0].item() == 1          # the rank still signalled its peer and moved on
    with pytest.raises(scmx._lib.ScmxError, match="peer barrier"):
        L.check_status()
    assert status[0].item() == 0                                  # check_status() clears the word
    # the context is still usable and a barrier of a world of one completes at once
    L.call("scmx_peer_barrier", peers, 0, 1, L.ptr(epoch), L.ptr(status), L.stream())
    torch.cuda.synchronize()
    L.check_status()
    assert epoch.item() == 2


def test_wait_limit_range(scmx):
    L = scmx._lib
    assert L.lib().scmx_set_wait_limit_ns(10) == -1
    assert L.lib().scmx_set_wait_limit_ns(2_000_000_000) == 0


def test_decode_step_wait_runs_out_and_reports(scmx):
    """Eight CTAs attend to 400,000 positions each (about 2 ms) while all others wait for the attention output with a limit of 1 us, looked at every 256 turns of 40 ns or
    more: the kernel returns, names the row of the first layer, and the next step on the same scratch has the chain's bits."""
    mod = lambda n: importlib.import_module(scmx.__name__ + "." + n)      # noqa: E731
    HM, FQ, DEC, L = mod("host_model"), mod("fused_qwen3"), mod("decode"), scmx._lib
    held, capacity = 400_000, 400_008
    model = HM.CausalLM(HM.ModelArgs(1024, 1024, 2, 8, 8, 128, 1e-6, 1e6, 512, True)).init_random(seed=5, scale=0.05).cuda()
    fused = FQ.FusedQwen3(model, FQ.pack_model(model, on_device=True))
    chain, mk = DEC.DecodeQwen3(fused, persistent=False), DEC.DecodeQwen3(fused, persistent=True)
    g = torch.Generator(device="cuda").manual_seed(5)
    long, short = fused.make_cache(capacity), [fused.make_cache(16) for _ in range(2)]
    for c in long:
        c.k.normal_(generator=g), c.v.normal_(generator=g)
        c.offset = held
    tok = torch.tensor([[7]], device="cuda")
    few = mk.attn.nsplit
    mk.attn.nsplit = 1
    mk.step(tok, long)                                # in time with the limit as it is
    mk.check_status()
    L.call("scmx_set_wait_limit_ns", 1000)
    try:
        t0 = time.perf_counter()
        mk.step(tok, long)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    finally:
        L.call("scmx_set_wait_limit_ns", 2_000_000_000)
    assert dt < 1.0
    assert int(mk._mk["status"].item()) == 1002
    with pytest.raises(L.ScmxError, match="layer 0 waiting for its attention output"):
        mk.check_status()
    # the same scratch again: the abort word and the epochs of the step that gave up are gone
    mk._mk["status"].zero_()
    scratch = mk._mk["scratch"]
    mk._mk, old = None, mk._mk
    mk._persistent_state(short[1])["scratch"] = scratch
    assert old["scratch"][:8].view(torch.int32)[1].item() == 1
    mk.attn.nsplit = 1
    for c, d in zip(*short):
        c.k.zero_(), c.v.zero_(), d.k.zero_(), d.v.zero_()
    chain.attn.nsplit = 1
    for _ in range(2):
        assert torch.equal(chain.step(tok, short[0]), mk.step(tok, short[1]))
    mk.check_status()
    mk.attn.nsplit = chain.attn.nsplit = few
