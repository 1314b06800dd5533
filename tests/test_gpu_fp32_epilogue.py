"""The 3xBF16 GEMM's C += AB epilogue: tiles of one, two and more accumulator
chunks, ragged last rows and columns, and grids in which a CTA computes several
tiles. The operands are small integers, so every sum is exact in FP32.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", ["128", "256"])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (33, 64, 129), (160, 65, 287), (129, 130, 257), (127, 1000, 31),
                                   (2573, 40, 4867)])
def test_exact_update(phpc, torch_cuda, monkeypatch, bn, m, k, n):
    torch = torch_cuda
    monkeypatch.setenv("PHPC_F32_BN", bn)
    monkeypatch.setenv("PHPC_F32_KSPLIT", "1")
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randint(-8, 9, (m, k), device="cuda", generator=g).float()
    B = torch.randint(-8, 9, (k, n), device="cuda", generator=g).float()
    exact = A.double() @ B.double()
    ws = phpc.bf16x3_workspace_bytes(m, k, n)
    W = torch.empty(ws, dtype=torch.uint8, device="cuda")
    for pad in (0, 3):
        C0 = torch.randint(-99, 100, (m + 1, n + pad), device="cuda", generator=g).float()
        C = C0.clone()
        phpc.sgemm_bf16x3_dev(m, k, n, A, k, B, n, C[:m, :n], n + pad, W, ws)
        torch.cuda.synchronize()
        assert phpc.device_status() == 0
        assert torch.equal(C[:m, :n].double(), C0[:m, :n].double() + exact)
        assert torch.equal(C[:, n:], C0[:, n:]) and torch.equal(C[m], C0[m])  # nothing outside the block


@pytest.mark.parametrize("m,k,n", [(300, 94, 500), (1500, 448, 1500), (2100, 448, 1500), (129, 500, 128), (129, 500, 129),
                                   (132, 1200, 268), (611, 900, 279), (250, 600, 900)])
def test_tile_width_same_bits(phpc, torch_cuda, monkeypatch, m, k, n):
    """Both sides of the rules for 128-wide tiles (tiles that all run at once
    with K unsplit or split, n <= 128): the bits of the 256-wide tile."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randn((m, k), device="cuda", generator=g)
    B = torch.randn((k, n), device="cuda", generator=g)
    C0 = torch.randn((m, n), device="cuda", generator=g)
    ws = phpc.bf16x3_workspace_bytes(m, k, n)
    W = torch.empty(ws, dtype=torch.uint8, device="cuda")
    outs = []
    for bn in (None, "256", "128"):
        if bn:
            monkeypatch.setenv("PHPC_F32_BN", bn)
        C = C0.clone()
        phpc.sgemm_bf16x3_dev(m, k, n, A, k, B, n, C, n, W, ws)
        outs.append(C)
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
