"""The training step's kernels at the edges of their tiles: batches whose rows
per partial sum leave a remainder of the 32-row stage, and the GEMM's gate at a
pitch and base that are not multiples of 16 bytes.

Bars: gradients as in test_gpu_surrogate.py (relative L2 below 1e-2, cosine
above 0.9999 per parameter block, against the float64 restatement that rounds
to BF16 where the GPU stores BF16); the gate exactly equal to the aligned one,
the same values being multiplied.
"""
import numpy as np
import pytest
import torch

import mlp_ref

pytestmark = pytest.mark.gpu

BLOCKS = np.cumsum([0, 256 * 4, 256, 65536, 256, 65536, 256, 65536, 256, 16 * 256, 16])


@pytest.mark.parametrize("rows", [128, 2176, 4224])
def test_gradients_at_stage_remainders(grrt, need_gpu, rows):
    S = grrt.Surrogate(1)
    p = mlp_ref.random_params(7).astype(np.float32)
    S.set_params(p)
    X, Y = (a.astype(np.float32) for a in mlp_ref.random_batch(8, rows))
    _, g = S.gradients(X, Y)
    _, want = mlp_ref.loss_and_grads(p.astype(np.float64), X, Y, bf=True)
    for lo, hi in zip(BLOCKS[:-1], BLOCKS[1:]):
        a, b = g[lo:hi].astype(np.float64), want[lo:hi]
        nb = np.linalg.norm(b)
        assert np.linalg.norm(a - b) < 1e-2 * nb and a @ b > 0.9999 * np.linalg.norm(a) * nb, (lo, hi)


@pytest.mark.parametrize("pitch,offset", [(256, 1), (257, 0), (258, 3)])
def test_gate_at_any_alignment(grrt, need_gpu, pitch, offset):
    M, N, K = 300, 256, 128
    gen = torch.Generator(device="cuda").manual_seed(3)
    A = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    B = torch.randn(N, K, device="cuda", generator=gen).bfloat16()
    z = torch.randn(M, N, device="cuda", generator=gen)
    store = torch.zeros(M * pitch + offset, device="cuda")
    store[offset:].view(M, pitch)[:, :N] = z

    def run(gate, ld):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        rc = grrt.lib().grrt_surrogate_gemm_bf16(A.data_ptr(), K, B.data_ptr(), K, M, N, K, 1, None, gate, ld, 0, None,
                                                 N, out.data_ptr(), N, None)
        assert rc == 0
        return out

    assert torch.equal(run(z.data_ptr(), N), run(store.data_ptr() + 4 * offset, pitch))
