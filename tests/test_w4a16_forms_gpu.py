"""Every tile form of the dense W4A16 contraction on the same weights: the bits of a row do not depend on the form, on
the layout of the weights or on the rows beside it.  Which form a call runs on is read from its observation, so that a
change of the selection rule cannot leave a form untested unnoticed (the sizes are for a GPU of 148 SMs)."""
import pytest
import torch

import intent_b200 as ib
import oracle
from intent_b200 import prelayout
from intent_b200.runtime import native
from conftest import max_abs_rel

pytestmark = pytest.mark.gpu

PAIRS, SINGLE = "w4a16_gemm_pair_kernel CTA pairs, 512x256", "w4a16_gemm_kernel single CTA, "
ROWS = {     # columns: rows of a call -> the form it runs on; the last row tile is ragged in every one
    4104: {77: SINGLE + "128x32", 129: SINGLE + "128x64", 500: SINGLE + "128x128", 600: SINGLE + "128x256",
           1100: PAIRS, 4100: SINGLE + "256x256"},
    # 600 rows: one tile per pair; 1100 rows: more tiles than pairs
    8200: {17: SINGLE + "128x64", 129: SINGLE + "128x128", 300: SINGLE + "128x256", 600: PAIRS, 1100: PAIRS,
           4100: SINGLE + "256x256"},
}


@pytest.mark.parametrize("dtype,zero_point,group,K,N", [
    (torch.bfloat16, 8, 32, 1056, 4104),                     # half a k block at the end, two scale rows per block
    (torch.float16, "twos_complement", 64, 1088, 8200),      # 17 k blocks
    (torch.bfloat16, "twos_complement", 128, 1152, 8200),    # 18 k blocks
    (torch.float16, 8, 32, 160, 4104),                       # fewer k blocks than sets of dequantiser warps
])
def test_every_form_gives_the_same_bits(cuda_device, dtype, zero_point, group, K, N):
    x, p, s = ib.workloads.w4a16_inputs(4100, K, N, dtype=dtype, group_size=group, seed=K)
    constants = {"GROUP_SIZE": group, "ZERO_POINT": zero_point, "KERNEL": "gemm",
                 "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"}
    target = ib.B200Target(0)
    plain = ib.compile(ib.programs.weight_only_int4_matmul, target=target, constexprs=constants)
    tiled = ib.compile(ib.programs.weight_only_int4_matmul, target=target,
                       constexprs=dict(constants, WEIGHT_LAYOUT="tiled"))
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    td = prelayout.tile(pd).tensor
    whole = plain.run(xd, pd, sd)
    for rows, kernel in ROWS[N].items():
        part = xd[:rows].contiguous()
        for artifact, weight in ((plain, pd), (tiled, td)):
            out = artifact.run(part, weight, sd)
            assert artifact.observation.kernel.startswith(kernel), (rows, artifact.observation.kernel)
            assert torch.equal(out, whole[:rows]), (rows, kernel)
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0
    # against the oracle that rounds the weight as the kernels do (the tolerances of test_w4a16_gemm_gpu.py)
    rounded = oracle.weight_only_int4_matmul_rounded(x[:1100], p, s, group_size=group,
                                                     zero_point=8 if zero_point == 8 else None)
    assert max_abs_rel(whole[:1100].cpu(), rounded) <= (2e-3 if dtype == torch.float16 else 1.6e-2)
