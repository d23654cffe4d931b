"""The GEMM's choice between its shapes where K is long: 32-column tiles while they are all resident, 128-column
tiles beyond (many outputs, or many splits). Both add an output's products in the same order, so an output among
many has the bits it has among few; and the tolerance of tests/test_gpu_gemm.py against fp32."""
import pytest

from test_gpu_gemm_shapes import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64 * 8, 64 * 9 + 8, 64 * 17, 4096])
@pytest.mark.parametrize("M,N", [(128 * 37, 128), (128 * 37 + 1, 128), (130, 128 * 19), (1000, 1000)])
def test_many_outputs(M, N, K):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    Bt = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    C = run(A, Bt)
    ref = A.double() @ Bt.double().T
    assert (C.double() - ref).abs().max().item() <= 1e-4 * ref.abs().max().item()
    assert torch.equal(C[:128, :32], run(A[:128].contiguous(), Bt[:32].contiguous()))
    assert torch.equal(C[-3:, -8:], run(A[-3:].contiguous(), Bt[-8:].contiguous()))


@pytest.mark.parametrize("splits", [36, 37, 38])
def test_many_splits(splits):
    import torch

    g = torch.Generator(device="cuda").manual_seed(splits)
    K = 64 * 9 * splits
    A = torch.randn(100, K, device="cuda", generator=g).to(torch.bfloat16)
    Bt = torch.randn(128, K, device="cuda", generator=g).to(torch.bfloat16)
    C = run(A, Bt, splits)
    ref = A.double() @ Bt.double().T
    assert (C.double() - ref).abs().max().item() <= 1e-4 * ref.abs().max().item()
    assert torch.equal(C[:, :32], run(A, Bt[:32].contiguous(), splits))
