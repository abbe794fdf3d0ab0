"""The int8 kernel on lone CTAs (128 x 256 tiles) and on CTA pairs (256 x 256 tiles): edges of the tiles in rows,
columns and k, exact integers.  Which of the two a call runs on is read from its observation."""
import pytest
import torch

import intent_b200 as ib
import oracle
from oracle.packed import unpack_w4a8

pytestmark = pytest.mark.gpu


LONE, PAIRS = "i8_gemm_kernel 128x256 tiles", "i8_gemm_kernel CTA pairs"


def _operands(M, K, N):
    g = torch.Generator().manual_seed(M)
    a = torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-128, 128, (K, N), generator=g, dtype=torch.int8)
    return a, b, torch.randint(-1000, 1000, (N,), generator=g, dtype=torch.int32)


def _run(device, a, b, bias):
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    out = torch.full((a.shape[0], b.shape[1]), -1, dtype=torch.int32, device=device)
    artifact(a.to(device), b.to(device), bias.to(device), out)
    torch.cuda.synchronize()
    artifact.check()
    return out.cpu(), artifact.observation.kernel


@pytest.mark.parametrize("M,K,N", [(129, 16, 16), (256, 128, 256), (257, 144, 272), (385, 1040, 528), (2050, 256, 4112),
                                   (6200, 10832, 528)])     # (the last: two bands of the tile walk)
def test_lone_tiles_are_exact(cuda_device, M, K, N):
    a, b, bias = _operands(M, K, N)
    out, kernel = _run(cuda_device, a, b, bias)
    assert kernel.startswith(LONE)
    assert torch.equal(out, oracle.gemm_i8_exact_f64(a, b, bias))


@pytest.mark.parametrize("M,K,N", [
    (129, 4112, 1040),      # the second CTA of the pair holds one row; 16 k at the end; 16 columns in the last tile
    (1400, 1040, 4112),     # more tiles than pairs, an odd count of 128-row tiles
    (4500, 2064, 528),      # more than 4096 rows, all in one band of the tile walk
    (8200, 8192, 528),      # 64 MB of A: three bands, the last of one row tile
])
def test_pair_tiles_are_exact(cuda_device, M, K, N):
    a, b, bias = _operands(M, K, N)
    out, kernel = _run(cuda_device, a, b, bias)
    assert kernel.startswith(PAIRS)
    assert torch.equal(out, oracle.gemm_i8_exact_f64(a, b, bias))


@pytest.mark.parametrize("M,K,N,kernel", [      # activation rows, k, weight rows (the rows of the product)
    (4112, 1056, 1400, PAIRS),    # both operands ragged, more tiles than pairs
    (1168, 6496, 816, PAIRS),     # one tile per pair; the rows of B share lines of the L2
    (16, 2048, 4112, PAIRS),      # sixteen columns, many row tiles
    (1168, 6528, 816, LONE),      # the rows of B on lines of their own
    (272, 7168, 9400, LONE),      # 64 MB of A: three bands of the tile walk
    (48, 2080, 816, LONE),        # little of B to share
])
def test_second_operand_k_major(cuda_device, M, K, N, kernel):
    """The packed programs hand their decoded weights over as the first operand and the activations as B [N, K]."""
    g = torch.Generator().manual_seed(3)
    activation = torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8)
    packed = torch.randint(0, 256, (N, K // 2), generator=g, dtype=torch.uint8)
    artifact = ib.compile(ib.programs.w4a8_packed_matmul, target=ib.B200Target(0))
    out = artifact.run(activation.to(cuda_device), packed.to(cuda_device))        # [N, M]
    torch.cuda.synchronize()
    artifact.check()
    assert artifact.observation.kernel.startswith(kernel)
    assert torch.equal(out.cpu(), oracle.gemm_i8_exact_f64(unpack_w4a8(packed), activation.T))


@pytest.mark.parametrize("M,K,N,kernel", [
    (128, 8192, 8192, LONE),                                 # one row tile
    (512, 1024, 2048, LONE), (512, 4096, 2048, PAIRS),       # too few k blocks to earn the pair launch back, and enough
    (129, 3072, 1024, LONE), (129, 8192, 1024, PAIRS),       # the same for eight tiles
    (2050, 1024, 2048, LONE), (2048, 1024, 2048, PAIRS),     # an odd row tile, many row tiles
    (135, 2240, 4480, LONE), (135, 2240, 4496, PAIRS),       # rows of B on lines of their own, and sharing them
    (3934, 576, 3664, LONE), (1840, 1536, 7520, LONE),       # several waves: few k blocks; a narrow last column
])
def test_short_walks_run_on_lone_tiles(cuda_device, M, K, N, kernel):
    a, b, bias = (t.to(cuda_device) for t in _operands(M, K, N))
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    artifact.run(a, b, bias)
    torch.cuda.synchronize()
    assert artifact.observation.kernel.startswith(kernel)
