"""Row strides of the operand planes.

Plane rows are padded to whole sectors or lines, and a grouped plan keeps a
store map per problem; a workspace that only holds rows padded to 16 bytes
(and no store maps) is accepted too, and gives the same bits; one byte less is
refused.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 13


def _up(x, to):
    return -(-x // to) * to


def _tail(m, k, n, planes, ld):
    """Bytes of the A and B planes with row stride ld, each aligned to 256."""
    return _up(planes * m * ld * 2, 256) + _up(planes * n * ld * 2, 256)


def _ld(k):
    return _up(k, 64 if k >= 256 else 16)


def _small(full, shapes, planes):
    """The workspace with 16-byte rows, from the one with padded rows."""
    return full - sum(_tail(m, k, n, planes, _ld(k)) - _tail(m, k, n, planes, _up(k, 8)) for m, k, n in shapes)


def _inputs(torch, m, k, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = [torch.randn(s, dtype=dtype, device="cuda", generator=g) for s in ((m, k), (k, n), (m, n))]
    return x


SHAPES = [(70, 13, 30), (130, 250, 257), (129, 264, 40), (200, 1000, 300)]


@pytest.mark.parametrize("kind", ["split", "f32"])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_small_workspace_same_bits(phpc, torch_cuda, kind, m, k, n):
    torch = torch_cuda
    if kind == "split":
        A, B, C = _inputs(torch, m, k, n, torch.float64)
        full, planes = phpc.ozaki2_workspace_bytes(m, k, n, Q), Q

        def call(c, w, size):
            phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, c, n, Q, w, size)
    else:
        A, B, C = _inputs(torch, m, k, n, torch.float32)
        full, planes = phpc.bf16x3_workspace_bytes(m, k, n), 3

        def call(c, w, size):
            phpc.sgemm_bf16x3_dev(m, k, n, A, k, B, n, c, n, w, size)
    small = _small(full, [(m, k, n)], planes)
    W = torch.full((full,), 0xFF, dtype=torch.uint8, device="cuda")  # NaN in every plane element not written
    C1, C2 = C.clone(), C.clone()
    call(C1, W, full)
    W.fill_(0xFF)
    call(C2, W, small)
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    assert torch.equal(C1, C2) and bool(torch.isfinite(C1).all())
    ref = C.double() + A.double() @ B.double()
    err = float((C1.double() - ref).norm() / ref.norm())
    assert err <= (1e-14 if kind == "split" else 2e-6)
    with pytest.raises(phpc.PhpcError) as e:
        call(C2, W, small - 1)
    assert e.value.code == 6


def test_grouped_small_workspace_same_bits(phpc, torch_cuda):
    torch = torch_cuda
    mats = [_inputs(torch, m, k, n, torch.float64) for m, k, n in SHAPES]
    outs = []
    maps = _up(128 * len(SHAPES), 256)
    for size_of in (lambda full: full, lambda full: _small(full, SHAPES, Q) - maps):
        Cs = [c.clone() for _, _, c in mats]
        probs = [(m, k, n, a, k, b, n, c, n) for (m, k, n), (a, b, _), c in zip(SHAPES, mats, Cs)]
        size = size_of(phpc.GroupedPlan.workspace_bytes(probs, 0, moduli=Q))
        W = torch.full((size + 256,), 0xFF, dtype=torch.uint8, device="cuda")
        plan = phpc.GroupedPlan(probs, 0, W, size, moduli=Q)
        plan.graph_launch()
        torch.cuda.synchronize()
        assert phpc.device_status() == 0
        plan.close()
        outs.append(Cs)
        last = size, probs, W
    for x, y in zip(*outs):
        assert torch.equal(x, y)
    size, probs, W = last
    with pytest.raises(phpc.PhpcError) as e:
        phpc.GroupedPlan(probs, 0, W, size - 1, moduli=Q)
    assert e.value.code == 6
