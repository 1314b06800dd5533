"""Calls whose kernels come up while the one before them finishes.

Back-to-back calls on one workspace, each reading what the last one wrote (C of
one call is A of the next), on the default stream, on a stream of their own
and replayed from a captured graph: the same bits as calls with a wait after
each. Shapes cover the shared launches (K <= 1024), the merge kernel between
scan and split, two streams, CTA pairs and the K-split FP32 GEMM.
"""
import pytest

pytestmark = pytest.mark.gpu

Q = 13


def _chain(phpc, torch, kind, n, mats, outs, W, size, stream, wait):
    """outs[i] += outs[i - 1] @ mats[i], from a fixed outs[0]."""
    for i in range(1, len(outs)):
        if kind == "split":
            phpc.dgemm_ozaki2_dev(n, n, n, outs[i - 1], n, mats[i], n, outs[i], n, Q, W, size, stream)
        else:
            phpc.sgemm_bf16x3_dev(n, n, n, outs[i - 1], n, mats[i], n, outs[i], n, W, size, stream)
        if wait:
            torch.cuda.synchronize()


@pytest.mark.parametrize("kind,n", [("split", 130), ("split", 700), ("split", 1100), ("split", 2048), ("f32", 200),
                                    ("f32", 640)])
def test_chained_calls(phpc, torch_cuda, kind, n):
    torch = torch_cuda
    dtype = torch.float64 if kind == "split" else torch.float32
    size = phpc.ozaki2_workspace_bytes(n, n, n, Q) if kind == "split" else phpc.bf16x3_workspace_bytes(n, n, n)
    W = torch.zeros(size, dtype=torch.uint8, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n)
    mats = [torch.randn((n, n), dtype=dtype, device="cuda", generator=g) / n ** 0.5 for _ in range(6)]
    first = torch.randn((n, n), dtype=dtype, device="cuda", generator=g)

    def fresh():
        return [first.clone()] + [torch.zeros_like(first) for _ in mats[1:]]

    want = fresh()
    _chain(phpc, torch, kind, n, mats, want, W, size, torch.cuda.current_stream(), True)
    outs = fresh()
    _chain(phpc, torch, kind, n, mats, outs, W, size, torch.cuda.current_stream(), False)
    torch.cuda.synchronize()
    for a, b in zip(outs, want):
        assert torch.equal(a, b)
    own = torch.cuda.Stream()
    outs = fresh()
    torch.cuda.synchronize()
    _chain(phpc, torch, kind, n, mats, outs, W, size, own, False)
    own.synchronize()
    for a, b in zip(outs, want):
        assert torch.equal(a, b)
    outs = fresh()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=own):
        _chain(phpc, torch, kind, n, mats, outs, W, size, own, False)
    for _ in range(2):
        for o in outs[1:]:
            o.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(outs, want):
            assert torch.equal(a, b)
    assert phpc.device_status() == 0
