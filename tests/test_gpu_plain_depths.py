"""The plain FP64 GEMM's ring depth on each of its tiles.

(test_gpu_pipeline_depth.py sweeps the depth under PHPC_DMMA_TILE = 64 and 128,
which both stand for the 32 x 32 tile.) 8 x 16 tiles are the scalar pipe's
only; every depth, tile and pipe gives the same bits.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(250, 514, 302), (70, 17, 40), (129, 96, 33)])
@pytest.mark.parametrize("tile", ["8", "16", "32"])
def test_every_depth_same_bits(phpc, torch_cuda, monkeypatch, tile, m, k, n):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    lda, ldb = k + (k & 1), n + (n & 1)
    A = torch.randn((m, lda), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((k, ldb), dtype=torch.float64, device="cuda", generator=g)
    C0 = torch.randn((m, n), dtype=torch.float64, device="cuda", generator=g)
    ref = C0.clone()
    phpc.dgemm_dmma_dev(m, k, n, A, lda, B, ldb, ref, n, 1, 1, 256)
    monkeypatch.setenv("PHPC_DMMA_TILE", tile)
    for pipe in ("dfma",) if tile == "8" else ("dfma", "dmma"):
        monkeypatch.setenv("PHPC_FP64_PIPE", pipe)
        for stages in ("2", "3", "4", "5", "6"):
            monkeypatch.setenv("PHPC_DMMA_STAGES", stages)
            C = C0.clone()
            phpc.dgemm_dmma_dev(m, k, n, A, lda, B, ldb, C, n, 1, 1, 256)
            torch.cuda.synchronize()
            assert torch.equal(C, ref), (pipe, stages)
    assert phpc.device_status() == 0
