"""W4A16 calls of few rows on column tiles of 64 and 32 columns: edges of the tile in rows, columns and k, and
fewer k blocks than there are sets of dequantiser warps.  (All forms side by side: test_w4a16_forms_gpu.py.)"""
import pytest
import torch

import intent_b200 as ib
import oracle
from conftest import max_abs_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,M,K,N,group", [
    (torch.float16, 17, 64, 8, 64),            # one k block, one tile of eight columns
    (torch.bfloat16, 128, 96, 40, 32),         # half a k block at the end, two scale rows per block
    (torch.float16, 33, 1088, 1000, 64),       # 17 k blocks, one more than the sets of the narrowest tile
    (torch.bfloat16, 77, 2048, 4104, 128),
    (torch.bfloat16, 129, 1024, 2056, 128),    # a second row tile of one row
    (torch.float16, 511, 1152, 2048, 128),
])
def test_narrow_tiles_give_the_bits_of_the_wide_ones(cuda_device, dtype, M, K, N, group):
    """Up to K = 2048 every tile form adds the k blocks in the same order, so a row's bits do not depend on how many rows
    the call has (longer K: test_w4a16_tmem_gpu.py; 4096 rows take a wider tile, or the same one where there are only 8 or 40 columns); the tolerances against
    the oracle are those of the wide tiles (test_w4a16_gemm_gpu.py)."""
    x, p, s = ib.workloads.w4a16_inputs(4096, K, N, dtype=dtype, group_size=group, seed=M)
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": group, "ZERO_POINT": 8,
                                      "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"})
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    whole = artifact.run(xd, pd, sd)
    out = artifact.run(xd[:M].contiguous(), pd, sd)
    assert artifact.observation.kernel.startswith(f"w4a16_gemm_kernel single CTA, 128x{64 if M == 511 else 32} ")
    torch.cuda.synchronize()
    artifact.check()
    assert torch.equal(out, whole[:M])
    rounded = oracle.weight_only_int4_matmul_rounded(x[:M], p, s, group_size=group, zero_point=8)
    assert max_abs_rel(out.cpu(), rounded) <= (2e-3 if dtype == torch.float16 else 1.6e-2)
