"""Short calls at head_dim 16 and 32 stay on the shape-generic kernels, which are faster there."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _C, flash


@pytest.mark.parametrize("D", [16, 32])
def test_backward_workspace(built_lib, D):
    need = lambda M, N, p=0.0: _C.call("fa_flash_bwd_workspace_bytes")(
        _C.pack_shape(torch.bfloat16, 2, 8, 8, M, N, D, True, 0.1, p))
    for M, N in ((64, 64), (160, 160), (32, 512), (512, 32)):
        assert need(M, N) == 0
    assert need(64, 64, 0.1) == 0 and need(96, 96, 0.1) > 0
    for M, N in ((192, 192), (64, 1024), (1000, 700)):
        assert need(M, N) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,M,N,D,p", [(2, 8, 300, 300, 32, 0.0), (2, 8, 300, 1024, 16, 0.0), (2, 8, 128, 128, 32, 0.1)])
def test_forward(B, H, M, N, D, p):
    """The same bits as with the generic kernels asked for."""
    q, k, v = (torch.randn(B, H, n, D, device="cuda", dtype=torch.bfloat16) for n in (M, N, N))
    run = lambda: flash._forward(q, k, v, True, D ** -0.5, p, 3, 5)
    with _C.kernel_family("generic"):
        want = run()
    for x, y in zip(run(), want):
        assert torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,D", [(500, 500, 32), (1000, 1000, 16)])
def test_piecewise_and_total(M, N, D):
    q1, k1, q2, k2, v = (torch.randn(2, 4, n, D, device="cuda", dtype=torch.float16) for n in (M, N, M, N, N))
    lse = torch.zeros(2, 4, M, device="cuda")
    run = lambda: (fa.piecewise_attention(q1, k1, q2, k2, v, 100, True), flash._total_attention(q1, k1, lse, True, D ** -0.5))
    with _C.kernel_family("generic"):
        want = run()
    for x, y in zip(run(), want):
        assert torch.equal(x, y)
