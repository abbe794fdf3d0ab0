"""The route alignment in one launch against the four programs that it stands for (exact integers)."""
import pytest
import torch

import intent_b200 as ib
from intent_b200.moe import MoEAlignment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,given,experts,block", [(1, 1, 1, 128), (40, 33, 8, 128), (1000, 1000, 3, 16),
                                                        (2049, 2049, 100, 256), (300, 300, 8192, 128)])
def test_one_launch_equals_the_stages(cuda_device, tokens, given, experts, block):
    g = torch.Generator().manual_seed(tokens + experts)
    ids = torch.randint(-1, experts + 1, (given, 2), generator=g, dtype=torch.int32)     # ids outside the table too
    alignment = MoEAlignment.build(tokens=tokens, top_k=2, experts=experts, block_size=block, target=ib.B200Target(0))
    ids = ids.to(cuda_device)
    routes, blocks, total = alignment.run(ids)
    counters, staged = alignment._buffers(cuda_device)
    staged, staged_blocks, staged_total = alignment.run_into(ids, counters[:experts], counters[experts:], staged)
    torch.cuda.synchronize()
    assert torch.equal(total, staged_total)
    assert torch.equal(routes, staged)
    used = int(total) // block
    assert torch.equal(blocks[:used], staged_blocks[:used])
