"""The residue GEMM with K split over a cluster of CTAs: residues are exact, so
every cluster size gives the unsplit product's bits, at shapes where the shares,
rows or columns are ragged, and writes nothing outside C's block.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", ["128", "256"])
@pytest.mark.parametrize("moduli", [8, 13])
@pytest.mark.parametrize("m,k,n", [(1, 65, 1), (129, 500, 257), (100, 1025, 130), (256, 1536, 256), (70, 4100, 301)])
def test_same_bits(phpc, torch_cuda, monkeypatch, bn, moduli, m, k, n):
    torch = torch_cuda
    monkeypatch.setenv("PHPC_OZAKI_BN", bn)
    monkeypatch.setenv("PHPC_CLUSTER", "1")
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randn((m, k), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g)
    C0 = torch.randn((m + 1, n + 3), dtype=torch.float64, device="cuda", generator=g)
    size = phpc.ozaki2_workspace_bytes(m, k, n, moduli)
    ref = None
    for split in ("1", "2", "3", "4", "5", "6", "7", "8", None):
        if split:
            monkeypatch.setenv("PHPC_RESIDUE_KSPLIT", split)
        else:
            monkeypatch.delenv("PHPC_RESIDUE_KSPLIT")
        W = torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda")
        C = C0.clone()
        phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, C, C.stride(0), moduli, W, size)
        torch.cuda.synchronize()
        assert phpc.device_status() == 0
        ref = C if ref is None else ref
        assert torch.equal(C, ref), split
    assert torch.equal(ref[:, n:], C0[:, n:]) and torch.equal(ref[m], C0[m])
    assert not torch.equal(ref[:m, :n], C0[:m, :n])


@pytest.mark.parametrize("m,k,n", [(128, 70, 128), (300, 300, 129), (124, 600, 1317), (600, 600, 400), (3000, 520, 100)])
def test_tile_width_same_bits(phpc, torch_cuda, monkeypatch, m, k, n):
    """Both sides of the rule for 128-wide tiles (n <= 128, units that all run
    at once): the bits of the 256-wide tile."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randn((m, k), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g)
    C0 = torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g)
    size = phpc.ozaki2_workspace_bytes(m, k, n, 13)
    W = torch.empty(size, dtype=torch.uint8, device="cuda")
    outs = []
    for bn in (None, "256", "128"):
        if bn:
            monkeypatch.setenv("PHPC_OZAKI_BN", bn)
        C = C0.clone()
        phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, C, n, 13, W, size)
        outs.append(C)
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
