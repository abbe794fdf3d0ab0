"""What an artifact keeps goes with its last reference, without a collection."""
import gc
import weakref

import pytest
import torch

import intent_b200 as ib

pytestmark = pytest.mark.gpu


def test_a_dropped_artifact_is_freed_at_once(cuda_device):
    x, p, s = ib.workloads.w4a16_inputs(1, 1024, 512, dtype=torch.float16, seed=0)
    args = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8})
    artifact.run(*args)
    assert artifact.observation.status == 0
    program = weakref.ref(artifact.runtime)
    gc.disable()
    try:
        del artifact
        assert program() is None
    finally:
        gc.enable()
