"""The int8 kernel on CTA pairs (256 x 256 tiles): edges of the pair tile in rows, columns and k, exact integers."""
import pytest
import torch

import intent_b200 as ib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(129, 16, 16), (256, 128, 256), (257, 144, 272), (385, 1040, 528), (2050, 256, 4112)])
def test_pair_tiles_are_exact(cuda_device, M, K, N):
    g = torch.Generator().manual_seed(M)
    a = torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-128, 128, (K, N), generator=g, dtype=torch.int8)
    bias = torch.randint(-1000, 1000, (N,), generator=g, dtype=torch.int32)
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    out = torch.full((M, N), -1, dtype=torch.int32, device=cuda_device)
    artifact(a.to(cuda_device), b.to(cuda_device), bias.to(cuda_device), out)
    torch.cuda.synchronize()
    artifact.check()
    # 16384 * 1040 < 2^24: the products and their sums are exact in f32
    expected = (a.float() @ b.float()).to(torch.int32) + bias
    assert torch.equal(out.cpu(), expected)
