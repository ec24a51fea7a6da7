"""The tcgen05 GEMM's gated epilogue where the last tile of 128 rows is not
full and the gate is not 16-byte aligned, against a float64 product (the bars of
test_gpu_surrogate_gemm.py: 1e-4 of the absolute sum + 1 through the gate)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 31, 33, 100, 127, 129, 300])
@pytest.mark.parametrize("N,offset,pitch", [(256, 0, 0), (256, 1, 0), (64, 0, 3), (16, 2, 1)])
def test_gate_with_a_part_tile(grrt, need_gpu, M, N, offset, pitch):
    K = 128
    g = torch.Generator(device="cuda").manual_seed(M + N + offset)
    A = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    B = (0.1 * torch.randn(N, K, device="cuda", generator=g)).bfloat16()
    ld = N + pitch
    store = torch.randn(offset + M * ld, device="cuda", generator=g)
    gate = store[offset:].view(M, ld)[:, :N]
    out = torch.full((M + 1, N), float("nan"), device="cuda")  # a row behind the last
    rc = grrt.lib().grrt_surrogate_gemm_bf16(A.data_ptr(), K, B.data_ptr(), K, M, N, K, 1, None,
                                             store.data_ptr() + 4 * offset, ld, 0, out.data_ptr(), N, None, N, None)
    assert rc == 0
    torch.cuda.synchronize()
    a, b, z = A.double(), B.double(), gate.double()
    s = torch.sigmoid(z)
    want = (a @ b.T) * s * (1 + z * (1 - s))
    assert bool(((out[:M].double() - want).abs() <= 1e-4 * (a.abs() @ b.abs().T + 1)).all())
    assert bool(out[M].isnan().all())
