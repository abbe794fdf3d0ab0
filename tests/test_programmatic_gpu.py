"""Programmatic launches: kernels of one program and of several start while the one ahead is still running, and must see what
that one wrote and leave alone what it still reads."""
import pytest
import torch

import intent_b200 as ib
import oracle
from intent_b200.moe import MoEW4A16FFN
from intent_b200.runtime import native

pytestmark = pytest.mark.gpu
TARGET = ib.B200Target(0)


def _packed(seed, M, K, N, per_byte):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=torch.int8),
            torch.randint(0, 256, (N, K // per_byte), generator=g, device="cuda", dtype=torch.uint8))


@pytest.mark.parametrize("program,per_byte,M,K,N", [
    ("bitnet_int2_matmul", 4, 1, 1024, 512),        # one kernel
    ("bitnet_int2_matmul", 4, 48, 1024, 512),       # expansion into the workspace, then the contraction
    ("w4a8_packed_matmul", 2, 48, 1024, 512),
])
def test_chains_of_packed_programs(cuda_device, program, per_byte, M, K, N):
    """Calls by turns on two inputs, whose expansions share one workspace, without a synchronisation: an expansion must not
    start to write while the contraction before it still reads."""
    artifact = ib.compile(getattr(ib.programs, program), target=TARGET)
    inputs = [_packed(seed, M, K, N, per_byte) for seed in (1, 2)]
    expected = [getattr(oracle, program)(*(t.cpu() for t in pair)) for pair in inputs]
    outs = [artifact.run(*inputs[i % 2]) for i in range(60)]
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out.cpu(), expected[i % 2]), i


def test_inputs_written_just_before(cuda_device):
    """The activation of the next call is the copy launched right before it."""
    artifact = ib.compile(ib.programs.bitnet_int2_matmul, target=TARGET)
    (a, packed), (b, _) = (_packed(seed, 4, 4096, 256, 4) for seed in (3, 4))
    expected = [oracle.bitnet_int2_matmul(t.cpu(), packed.cpu()) for t in (a, b)]
    buffer, outs = torch.empty_like(a), []
    for i in range(60):
        buffer.copy_((a, b)[i % 2])
        outs.append(artifact.run(buffer, packed))
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out.cpu(), expected[i % 2]), i


def test_layer_calls_in_a_row(cuda_device):
    """Routes, alignment, gather and both contractions of different inputs in a row give what each gives alone."""
    tokens, hidden, intermediate, experts = 96, 512, 256, 8
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=TARGET)
    cases = []
    for seed in (11, 12, 13):
        data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=seed)
        cases.append({k: v.to(cuda_device) for k, v in data.items()})

    def call(dev):
        ids, weights = layer.route(dev["logits"])
        return layer(dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"],
                     dev["down_scales"])

    alone = []
    for dev in cases:
        alone.append(call(dev))
        torch.cuda.synchronize()
    outs = [call(cases[i % 3]) for i in range(30)]
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out, alone[i % 3]), i


def test_the_overlap_switch_behind_other_kernels(cuda_device):
    """With the switch on a bandwidth call may ask for its weights while the call before it is running.  That call, when it
    is of another program, must not have started before the copy ahead of it wrote the weights."""
    K, N = 4096, 4096
    x, p, s = ib.workloads.w4a16_inputs(1, K, N, dtype=torch.bfloat16, seed=1)
    other = ib.workloads.w4a16_inputs(1, K, N, dtype=torch.bfloat16, seed=2)[1].to(cuda_device)
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    gemv = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0), constexprs={
        "GROUP_SIZE": 128, "ZERO_POINT": 8, "ACT_DTYPE": "bf16", "KERNEL": "gemv"})
    between = ib.compile(ib.programs.bitnet_int2_matmul, target=ib.B200Target(0))
    act = torch.ones((1, 256), dtype=torch.int8, device=cuda_device)
    codes = torch.ones((16, 64), dtype=torch.uint8, device=cuda_device)
    expected = gemv.run(xd, other, sd)
    weights, busy = pd.clone(), torch.randn((4096, 4096), device=cuda_device)
    library = native.library()
    try:
        assert library.intent_b200_w4a16_gemv_overlap(1) == 0
        for _ in range(50):
            weights.copy_(pd)
            busy @ busy
            weights.copy_(other)
            between.run(act, codes)
            assert torch.equal(gemv.run(xd, weights, sd), expected)
    finally:
        library.intent_b200_w4a16_gemv_overlap(0)
