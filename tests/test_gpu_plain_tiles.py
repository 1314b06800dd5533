"""The plain FP64 GEMM's tiles (8 x 16, 16 x 16 and 32 x 32) on both pipes.

Every output is summed over k in increasing order with one rounding per FMA
and added into C once, whatever the tile, pipe or SUMMA grid, so all variants
must agree bit for bit.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (15, 16, 17), (16, 17, 16), (33, 15, 31), (65, 300, 40), (250, 514, 302), (68, 200, 1617)])
@pytest.mark.parametrize("gw,gh", [(1, 1), (3, 2), (64, 64)])
def test_tiles_pipes_and_grids_same_bits(phpc, torch_cuda, monkeypatch, m, k, n, gw, gh):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m * k + n)
    lda, ldb, ldc = k + (k & 1) + 2, n + (n & 1) + 4, n + 3
    A = torch.randn((m, lda), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((k, ldb), dtype=torch.float64, device="cuda", generator=g)
    C0 = torch.randn((m, ldc), dtype=torch.float64, device="cuda", generator=g)
    outs = {}
    for tile in ("8", "16", "32", None):
        for pipe in ("dfma", "dmma"):
            monkeypatch.setenv("PHPC_FP64_PIPE", pipe)
            if tile:
                monkeypatch.setenv("PHPC_DMMA_TILE", tile)
            else:
                monkeypatch.delenv("PHPC_DMMA_TILE", raising=False)
            C = C0.clone()
            phpc.dgemm_dmma_dev(m, k, n, A, lda, B, ldb, C, ldc, gw, gh, 256)
            outs[tile, pipe] = C
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    first = outs["16", "dfma"]
    for key, C in outs.items():
        assert torch.equal(C, first), key
    assert torch.equal(first[:, n:], C0[:, n:])  # nothing beyond the n columns
    ref = C0[:, :n] + A[:, :k] @ B[:k, :n]
    # k roundings of at most 2^-53 of the running sum each, in both sums
    bound = 2 * (k + 1) * 2.0 ** -53 * (C0[:, :n].abs() + A[:, :k].abs() @ B[:k, :n].abs())
    assert bool(((first[:, :n] - ref).abs() <= bound).all())
