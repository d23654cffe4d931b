"""The GEMM's two shapes (few K slices: 128-column tiles, two stages; many:
32-column tiles, eight stages) around their edges, against a torch fp32
reference with the tolerance of tests/test_gpu_gemm.py; and that the split into
column tiles does not change an output's value (a column alone equals the
column among others)."""
import ctypes as C

import pytest

from test_gpu_gemm import _gemm, _ptr

pytestmark = pytest.mark.gpu


def run(A, Bt, splits=1):
    import torch

    M, K, N = A.shape[0], A.shape[1], Bt.shape[0]
    Cf = torch.full((M, N), float("nan"), device="cuda")
    part = torch.zeros((splits, M, N), device="cuda") if splits > 1 else None
    err = C.c_uint32(0)
    torch.cuda.synchronize()
    rc = _gemm()(_ptr(A), _ptr(Bt), _ptr(Cf), None, None, M, N, K, K, K, N, 0, splits, _ptr(part),
                 C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(err))
    assert rc == 0 and err.value == 0
    return Cf


# K in slices of 64: the shapes change at 8 slices a split; rings wrap at 2 and 8
@pytest.mark.parametrize("K", [8, 64, 128, 136, 64 * 7, 64 * 7 + 8, 64 * 8, 64 * 9, 64 * 15 + 24, 64 * 16, 64 * 17, 13800])
@pytest.mark.parametrize("M,N", [(128, 128), (8, 256), (130, 8), (128, 40)])
def test_shapes_match_fp32_reference(M, N, K):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    Bt = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    ref = A.double() @ Bt.double().T
    scale = ref.abs().max().item()
    for splits in (1, 3):
        out = run(A, Bt, splits)
        assert (out - ref).abs().max().item() <= 1e-4 * scale


def test_column_tiles_do_not_change_a_value():
    import torch

    g = torch.Generator(device="cuda").manual_seed(2)
    A = torch.randn(100, 4000, device="cuda", generator=g).to(torch.bfloat16)
    Bt = torch.randn(96, 4000, device="cuda", generator=g).to(torch.bfloat16)
    whole = run(A, Bt)
    for c in (0, 31, 32, 95):
        assert torch.equal(run(A, Bt[c : c + 1].contiguous())[:, 0], whole[:, c])
