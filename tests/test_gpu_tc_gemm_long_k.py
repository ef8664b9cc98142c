"""The persistent product at K on both sides of the line between many epilogue warps and a long
operand ring: the two variants against the fp32 product, ragged in M and N."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(40037, 512), (39001, 128)])
@pytest.mark.parametrize("K", [1664, 1672, 1728, 2056])
@pytest.mark.parametrize("act", [0, 1])
def test_tc_gemm_persistent_long_k(lib, cuda, M, N, K, act):
    import torch
    g = torch.Generator(device="cpu").manual_seed(M + N + K + act)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(cuda)
    B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(cuda)
    bias = (torch.randn(N, generator=g) * 0.1).to(cuda)
    out = torch.full((M, N), float("nan"), dtype=torch.float32, device=cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    rc = lib.cumf_tc_gemm(A.data_ptr(), B.data_ptr(), M, N, K, bias.data_ptr(), act, out.data_ptr(), 1, N, None,
                          status.data_ptr(), None)
    assert rc == 0, lib.cumf_last_error()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    exp = A.float() @ B.float().T + bias
    if act:
        exp = torch.nn.functional.gelu(exp, approximate="tanh")
    assert (out - exp).abs().max().item() <= 1e-4 * exp.abs().max().item() + 1e-6
