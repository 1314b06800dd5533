"""The two column scans of a grouped modular plan: batches below and above the
number of (column, 256-row chunk) units at which they change over, with columns
and chunks that fill neither a warp nor a slice of 32 rows, zero columns and
exponents that rise or fall all along: the single call's bits for each problem.
"""
import pytest

pytestmark = pytest.mark.gpu

Q = 13


@pytest.mark.parametrize("copies", [1, 400])
def test_same_bits_as_single(phpc, torch_cuda, copies):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(copies)
    kinds = []
    for m, k, n in [(3, 1, 1), (9, 31, 33), (5, 33, 31), (8, 257, 70), (2, 255, 5), (7, 1025, 40), (4, 600, 64)]:
        A = torch.randn((m, k), dtype=torch.float64, device="cuda", generator=g)
        B = torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g)
        steps = torch.arange(k, device="cuda").clamp(max=900).to(torch.int32)
        B[:, 0] = torch.ldexp(B[:, 0], steps - 400)
        if n > 4:
            B[:, 1] = torch.ldexp(B[:, 1], 300 - steps)
            B[:, 2] = 0
            B[: k // 2, 3] = 0
        C = torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g)
        want = C.clone()
        size = phpc.ozaki2_workspace_bytes(m, k, n, Q)
        W = torch.empty(size, dtype=torch.uint8, device="cuda")
        phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, want, n, Q, W, size)
        kinds.append((m, k, n, A, B, C, want))
    probs, outs = [], []
    for _ in range(copies):
        for m, k, n, A, B, C, want in kinds:
            c = C.clone()
            probs.append((m, k, n, A, k, B, n, c, n))
            outs.append((c, want))
    units = copies * sum(n * -(-k // 256) for _, k, n, *_ in kinds)
    assert units < 10000 or units > 160 * 300  # one side of the rule or the other on any device
    size = phpc.GroupedPlan.workspace_bytes(probs, 7, moduli=Q)
    W = torch.empty(size, dtype=torch.uint8, device="cuda")
    plan = phpc.GroupedPlan(probs, 7, W, size, moduli=Q)
    plan.run()
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    assert all(torch.equal(c, want) for c, want in outs)
    plan.close()
