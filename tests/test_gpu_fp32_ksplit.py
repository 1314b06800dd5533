"""The 3xBF16 GEMM with K split over a cluster of CTAs.

Every cluster size against the unsplit tile, at shapes where the shares, rows
or columns are ragged: the same product to within what the order of a few FP32
additions can change, exact where every sum is, and nothing outside C's block.
"""
import pytest

pytestmark = pytest.mark.gpu


def _call(phpc, torch, A, B, C, k):
    m, n = C.shape[0], B.shape[1]
    ws = phpc.bf16x3_workspace_bytes(m, k, n)
    W = torch.empty(ws, dtype=torch.uint8, device="cuda")
    phpc.sgemm_bf16x3_dev(m, k, n, A, A.stride(0), B, B.stride(0), C, C.stride(0), W, ws)
    torch.cuda.synchronize()
    assert phpc.device_status() == 0


@pytest.mark.parametrize("bn", ["128", "256"])
@pytest.mark.parametrize("m,k,n", [(1, 65, 1), (129, 70, 257), (130, 600, 500), (100, 2000, 130), (300, 129, 1000)])
def test_every_split(phpc, torch_cuda, monkeypatch, bn, m, k, n):
    torch = torch_cuda
    monkeypatch.setenv("PHPC_F32_BN", bn)
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randn((m, k), device="cuda", generator=g)
    B = torch.randn((k, n), device="cuda", generator=g)
    C0 = torch.randn((m, n + 3), device="cuda", generator=g)
    Ai = torch.randint(-8, 9, (m, k), device="cuda", generator=g).float()
    Bi = torch.randint(-8, 9, (k, n), device="cuda", generator=g).float()
    ref = C0[:, :n].double() + A.double() @ B.double()
    scale = C0[:, :n].double().abs() + A.double().abs() @ B.double().abs()
    exact = Ai.double() @ Bi.double()  # below 2^24: every FP32 sum is exact
    for split in ("1", "2", "3", "4", "5", "6", "7", "8", None):
        if split:
            monkeypatch.setenv("PHPC_F32_KSPLIT", split)
        else:
            monkeypatch.delenv("PHPC_F32_KSPLIT")
        C = C0.clone()
        _call(phpc, torch, A, B, C[:, :n], k)
        assert torch.equal(C[:, n:], C0[:, n:]), split
        err = float((C[:, :n].double() - ref).norm() / ref.norm())
        assert err <= 2e-6, (split, err)
        assert bool(((C[:, :n].double() - ref).abs() <= 2e-6 * scale).all()), split
        C = torch.zeros((m, n + 3), device="cuda")
        _call(phpc, torch, Ai, Bi, C[:, :n], k)
        assert torch.equal(C[:, :n].double(), exact), split
