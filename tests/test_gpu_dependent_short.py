"""Dependent launches that test_gpu_dependent_launch.py's square chains miss.

Its 2048 makes none (preparation joins a second stream and the GEMM is long).
Here: a short call whose preparation runs on two streams (K > 2560), so that
only the CRT is dependent, with K split in the GEMM; the same between calls
whose every launch is dependent; and CTA pairs with a short GEMM
(PHPC_CLUSTER = 2). Calls follow one another on one workspace, each reading
what the last one wrote, with and without waits and from a captured graph.
"""
import pytest

pytestmark = pytest.mark.gpu

Q = 13


def _run(phpc, torch, shapes, mats, outs, W, size, stream, wait):
    """outs[i] += outs[i - 1] @ mats[i - 1], shapes[i] = (m, k, n)."""
    for (m, k, n), B, A, C in zip(shapes, mats, outs, outs[1:]):
        phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, C, n, Q, W, size, stream)
        if wait:
            torch.cuda.synchronize()


@pytest.mark.parametrize("dims,cluster", [
    ([128, 4096, 128, 4096, 128], None),  # 128 x 4096 x 128 and 128 x 128 x 4096 in turn
    ([60, 2700, 90, 3000, 2600, 40], None),  # two streams three times, K = 2600 and 3000 in a row
    ([300, 300, 700, 260, 520], "2"),
])
def test_chain(phpc, torch_cuda, monkeypatch, dims, cluster):
    torch = torch_cuda
    if cluster:
        monkeypatch.setenv("PHPC_CLUSTER", cluster)
    m = dims[0]
    shapes = [(m, k, n) for k, n in zip(dims[1:], dims[2:])]
    size = max(phpc.ozaki2_workspace_bytes(*s, Q) for s in shapes)
    W = torch.zeros(size, dtype=torch.uint8, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(sum(dims))
    first = torch.randn((m, dims[1]), dtype=torch.float64, device="cuda", generator=g)
    mats = [torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g) / k ** 0.5 for _, k, n in shapes]

    def fresh():
        return [first.clone()] + [torch.zeros((m, n), dtype=torch.float64, device="cuda") for _, _, n in shapes]

    want = fresh()
    _run(phpc, torch, shapes, mats, want, W, size, torch.cuda.current_stream(), True)
    ref = first
    for B, C in zip(mats, want[1:]):
        ref = ref @ B
        assert float((C - ref).norm() / ref.norm()) < 1e-13
    own = torch.cuda.Stream()
    for stream in (torch.cuda.current_stream(), own):
        outs = fresh()
        torch.cuda.synchronize()
        for _ in range(3):
            torch.cuda.synchronize()  # the zeroing below is on another stream than the calls
            for o in outs[1:]:
                o.zero_()
            torch.cuda.synchronize()
            _run(phpc, torch, shapes, mats, outs, W, size, stream, False)
        torch.cuda.synchronize()
        for a, b in zip(outs, want):
            assert torch.equal(a, b)
    outs = fresh()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=own):
        _run(phpc, torch, shapes, mats, outs, W, size, own, False)
    for _ in range(2):
        for o in outs[1:]:
            o.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(outs, want):
            assert torch.equal(a, b)
    assert phpc.device_status() == 0
