"""GPU: the few-rows GEMM (K split over a cluster) at the edges of its tiles, stages and splits, against the fp32 oracle."""
import pytest
import torch

import oasr_b200 as ob
from oasr_b200 import fused
from oracle import ops as O

pytestmark = pytest.mark.gpu

# rows: one, below / at / over the A box sizes and the 128-row tile, the largest of the kernel's range and the first beyond;
# K: one block, a tail, one split, 2 / 4 / 8 splits, and slices that are no multiple of a stage
SHAPES = [(1, 32, 64), (7, 40, 80), (16, 512, 512), (33, 2048, 512), (64, 96, 1024), (65, 264, 1032), (128, 512, 2048), (129, 512, 2112),
          (300, 1024, 4096), (16, 512, 9728), (78, 512, 9728), (592, 5008, 1024), (2560, 512, 2048), (2561, 256, 2048)]


def _rand(shape, dtype, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_every_epilogue_matches_the_oracle(dtype, M, N, K):
    A, B, C = _rand((M, K), dtype, 1), _rand((N, K), dtype, 2, K ** -0.5), _rand((N,), dtype, 3)
    want = O.gemm(A, B, C)
    # one rounding of a value of a few units: half an ulp is 2^-9 (bf16), 2^-12 (fp16) of it, plus fp32 sums in another order
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    dev = [t.cuda() for t in (A, B, C)]
    torch.testing.assert_close(ob.gemm(*dev).float().cpu(), want, rtol=ulp, atol=1e-4)
    # swish by one tanh.approx (relative error 2^-11) before the rounding
    torch.testing.assert_close(ob.gemm_activation(*dev, 2).float().cpu(), want * torch.sigmoid(want), rtol=ulp + 2.0 ** -10, atol=1e-3)
    R = _rand((M, N), torch.float32, 4)
    torch.testing.assert_close(ob.gemm_residual_f32(R.cuda(), *dev, 0.5).cpu(), R + 0.5 * want, rtol=1e-4, atol=1e-4)
    if N % 64 == 0:
        glu = want[:, :N // 2] * torch.sigmoid(want[:, N // 2:])
        torch.testing.assert_close(ob.gemm_glu(*dev).float().cpu(), glu, rtol=ulp + 2.0 ** -10, atol=1e-3)


@pytest.mark.parametrize("M", [3, 128, 2560])
def test_duplicated_block(M):
    d, K = 256, 512
    A, B, C = (_rand(s, torch.bfloat16, i, 0.1).cuda() for i, s in enumerate([(M, K), (3 * d, K), (4 * d,)]))
    assert torch.equal(fused.gemm_dup_first(A, B, C, d), ob.gemm(A, torch.cat([B[:d], B]), C))


@pytest.mark.parametrize("N,K", [(2048, 512), (512, 2048), (512, 9728), (4096, 512), (4096, 1024)])   # the last two change kernels
def test_a_row_does_not_depend_on_its_batch(N, K):
    """Outputs of up to 512 columns stay on the kernel, unsplit products give the bits of the one that takes over: bit-identical
    rows from 1 row to the whole range."""
    A, B = _rand((2560, K), torch.bfloat16, 5).cuda(), _rand((N, K), torch.bfloat16, 6, K ** -0.5).cuda()
    full = ob.gemm(A, B)
    for m in (1, 17, 100, 700):
        assert torch.equal(ob.gemm(A[:m].contiguous(), B), full[:m])


@pytest.mark.parametrize("M,N,K", [(1, 512, 512), (100, 4096, 512), (700, 4096, 1024), (1500, 2048, 520), (2560, 520, 968)])
def test_unsplit_products_have_the_bits_of_the_persistent_kernel(M, N, K):
    """What lets a product change kernels with its rows: store, swish, GLU and fp32 residual against a forced tile width, which
    names the kernel of gemm.cu."""
    from oasr_b200 import tunables

    A, B, C = _rand((M, K), torch.bfloat16, 7).cuda(), _rand((N, K), torch.bfloat16, 8, K ** -0.5).cuda(), _rand((N,), torch.bfloat16, 9).cuda()
    R = _rand((M, N), torch.float32, 10).cuda()
    every = lambda: [ob.gemm(A, B, C), ob.gemm_activation(A, B, C, 2), ob.gemm_residual_f32(R, A, B, C, 0.5)] + (
        [ob.gemm_glu(A, B, C)] if N % 16 == 0 else [])
    by_size = every()
    try:
        tunables.set("gemm_bn", 128)
        forced = every()
    finally:
        tunables.set("gemm_bn", 0)
    assert ob.device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(by_size, forced))
