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


def _bound(device, M, K, N):
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=torch.float16, seed=1)
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8})
    return artifact, artifact.prepare(x.to(device), p.to(device), s.to(device))


def test_an_observation_is_of_its_launch(cuda_device):
    """The facts are put together when they are read: switches turned since the launch, and storage given back since,
    do not change or lose them."""
    library = ib.runtime.native.library()
    artifact, call = _bound(cuda_device, 1, 1024, 512)
    try:
        assert library.intent_b200_w4a16_gemv_warps(16) == 0
        call.launch()
    finally:
        library.intent_b200_w4a16_gemv_warps(0)
    assert call.observation.threads == artifact.observation.threads == 512
    call.launch()                                       # the same binding, by the built-in choice
    assert call.observation.threads == artifact.observation.threads == 1024

    artifact, call = _bound(cuda_device, 2048, 128, 4096)
    try:
        assert library.intent_b200_w4a16_gemm_pairs(0) == 0
        call.launch()
    finally:
        library.intent_b200_w4a16_gemm_pairs(1)
    torch.cuda.synchronize()
    del call
    torch.cuda.empty_cache()
    assert artifact.observation.kernel.startswith("w4a16_gemm_kernel single CTA")
    artifact, call = _bound(cuda_device, 2048, 128, 4096)
    call.launch()
    torch.cuda.synchronize()
    assert artifact.observation.kernel.startswith("w4a16_gemm_pair_kernel")
