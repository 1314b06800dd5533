"""The modular call's tile width where 128-wide units all run at once: 128, but
256 where the half as many wide ones are split along K much more finely.
(Shapes measured on both sides of the rule; the bits never depend on it.)"""
import ctypes as ct

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moduli,m,k,n,bn", [(8, 569, 2600, 178, 128), (8, 569, 3453, 178, 256), (8, 569, 6000, 178, 256),
                                             (8, 700, 3453, 300, 128), (13, 100, 3453, 700, 256), (13, 569, 3453, 178, 128),
                                             (13, 250, 4500, 500, 128), (13, 300, 300, 300, 128)])
def test_width_and_bits(phpc, torch_cuda, monkeypatch, moduli, m, k, n, bn):
    torch = torch_cuda
    cfg = (ct.c_int * 10)()
    monkeypatch.setenv("PHPC_MODULI", str(moduli))
    assert phpc.lib().phpc_tuning(m, k, n, cfg) == 0
    assert cfg[2] == bn
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    A = torch.randn((m, k), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g)
    size = phpc.ozaki2_workspace_bytes(m, k, n, moduli)
    W = torch.empty(size, dtype=torch.uint8, device="cuda")
    outs = []
    for width in (None, "128", "256"):
        if width:
            monkeypatch.setenv("PHPC_OZAKI_BN", width)
        C = torch.zeros((m, n), dtype=torch.float64, device="cuda")
        phpc.dgemm_ozaki2_dev(m, k, n, A, k, B, n, C, n, moduli, W, size)
        outs.append(C)
    torch.cuda.synchronize()
    assert phpc.device_status() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
