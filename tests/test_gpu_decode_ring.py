"""GPU: one decode ring used again and again: its events and views serve eager passes, a captured pass, passes on other streams that start while the last one still reads, and
sequences of other weights, with groups that do not divide the sequence, and the operand each product reads is the decoded weight (compared as integers)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group, count", [(1, 1), (1, 2), (1, 5), (2, 5), (3, 7)])
@pytest.mark.parametrize("overlap", [True, False])
def test_ring_serves_every_pass(scmx, group, count, overlap):
    S = scmx.sc_kernels
    g = torch.Generator(device="cuda").manual_seed(count)
    shapes = [(256, 512), (512, 256), (128, 1024)]

    def weights(first):
        seq = []
        for i in range(count):
            n, k = shapes[(first + i) % 3]
            c = torch.randint(-2 ** 31, 2 ** 31 - 1, (n * k // 8,), generator=g, device="cuda").to(torch.int32)
            seq.append((c, torch.randint(0, 256, (n, k // 128), generator=g, device="cuda").to(torch.uint8), None, n, k))
        return seq

    def read(seq, slow=False):
        ring.begin(seq)
        got = []
        for i in range(count):
            w = ring.weight(i)
            if slow:
                torch.cuda._sleep(200_000)                # 0.1 ms: the host is through with the pass before its reads have begun
            got.append(w.clone())
            ring.released(i)
        ring.end()
        return got

    ring = scmx.fused_dense.DecodeRing(1 << 17, "cuda", overlap, group)
    seqs = [weights(0), weights(1)]
    want = [[S.unpack_i8(c, b, n, k) for c, b, _, n, k in seq] for seq in seqs]
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    outs = [(read(seqs[0]), 0), (read(seqs[1]), 1)]
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        kept = read(seqs[1])
    graph.replay()
    torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), side, torch.cuda.current_stream()):      # no synchronization in between
        with torch.cuda.stream(stream):
            outs += [(read(seqs[0], True), 0), (read(seqs[1], True), 1)]
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for got, i in outs + [(kept, 1)]:
        assert all(torch.equal(a, b) for a, b in zip(got, want[i]))
