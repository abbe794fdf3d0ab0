"""MoE router / alignment (bit-exact) and the grouped int4 FFN (2e-2 * max|ref|)."""
import pytest
import torch

import intent_b200 as ib
import oracle
from intent_b200.moe import MoEAlignment, MoEW4A16FFN
from intent_b200.runtime import native
from conftest import load_golden, max_abs_rel

pytestmark = pytest.mark.gpu


def test_router_top2_bit_exact(cuda_device):
    logits = ib.workloads.moe_inputs(16384, 64, 64, 128, seed=0)["logits"]       # benchmark router input
    logits[5, 7] = logits[5, 40] = logits[5].max() + 1.0                         # exact tie: lower id first
    logits[9, :] = 0.5                                                           # all equal: ids 0, 1
    router = ib.compile(ib.programs.moe_route_top2, target=ib.B200Target(0))
    ids, weights = router.run(logits.to(cuda_device))
    torch.cuda.synchronize()
    ref_ids, ref_weights = oracle.moe_route_top2(logits)
    assert ids.dtype == torch.int32 and torch.equal(ids.cpu(), ref_ids)
    assert ids[5].tolist() == [7, 40] and ids[9].tolist() == [0, 1]
    weights = weights.cpu()
    if not torch.allclose(weights, ref_weights, rtol=2e-6, atol=0):
        # which rows, and which side is off: both lie within 3e-7 of 64 bits where they are sound
        exact = torch.softmax(logits.double(), dim=1).gather(1, ref_ids.long())
        away = ((weights - ref_weights).abs() / ref_weights).amax(dim=1)
        rows = away.argsort(descending=True)[:4].tolist()
        again = router.run(logits.to(cuda_device))[1].cpu()
        pytest.fail(f"{int((away > 2e-6).sum())} rows differ; the worst (row, kernel, oracle, 64 bits, kernel once more): " +
                    "; ".join(f"{r} {weights[r].tolist()} {ref_weights[r].tolist()} {exact[r].tolist()} {again[r].tolist()}"
                              for r in rows))
    g = load_golden("insertion_top_k")                                           # reference golden, k = 8 -> first two
    ids, _ = router.run(g["logits"].to(cuda_device))
    assert torch.equal(ids.cpu(), g["indices"][:, :2])


@pytest.mark.parametrize("tag", ["ref_pattern", "small"])
def test_alignment_matches_reference_golden(cuda_device, tag):
    g = load_golden(f"moe_align_{tag}")
    block, experts = int(g["block"]), int(g["experts"])
    tokens = g["topk_ids"].shape[0]
    alignment = MoEAlignment.build(tokens=tokens, top_k=2, experts=experts, block_size=block, target=ib.B200Target(0))
    ids = g["topk_ids"].to(cuda_device)
    sorted_ids, expert_blocks, total = alignment.run(ids)
    torch.cuda.synchronize()
    assert torch.equal(total.cpu(), g["total"])
    assert torch.equal(sorted_ids.cpu(), g["sorted_ids"])                       # stable order: no canonicalisation needed
    blocks = int(total) // block
    assert torch.equal(expert_blocks[:blocks].cpu(), g["expert_ids"])
    # prepared form: same results on relaunch, workspace reset included
    call = alignment.prepare(ids)
    call.compile()
    call.launch()
    call.launch()
    torch.cuda.synchronize()
    again, blocks_again, total_again = call.result()
    assert torch.equal(again, sorted_ids) and torch.equal(total_again, total)
    assert torch.equal(call.counts.cpu(), g["counts"]) and torch.equal(call.cursors.cpu(), g["counts"])


def test_alignment_benchmark_size_properties(cuda_device):
    """16384 tokens, 64 experts: equal to the oracle, every route appears once, spans are sorted."""
    logits = ib.workloads.moe_inputs(16384, 64, 64, 128, seed=0)["logits"]
    ids, _ = oracle.moe_route_top2(logits)
    alignment = MoEAlignment.build(tokens=16384, top_k=2, experts=64, block_size=128, target=ib.B200Target(0))
    sorted_ids, expert_blocks, total = alignment.run(ids.to(cuda_device))
    ref_sorted, ref_blocks, ref_total, _ = oracle.moe_align_block_size(ids, 128, 64)
    assert torch.equal(total.cpu(), ref_total) and torch.equal(sorted_ids.cpu(), ref_sorted)
    n = int(total) // 128
    assert torch.equal(expert_blocks[:n].cpu(), ref_blocks[:n])
    real = sorted_ids[sorted_ids < 32768]
    assert real.numel() == 32768 and torch.equal(torch.sort(real).values.cpu(), torch.arange(32768, dtype=torch.int32))


def _ffn_case(tokens, hidden, intermediate, experts, dtype, seed):
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=dtype, seed=seed)
    ids, weights = oracle.moe_route_top2(data["logits"])
    return data, ids, weights


@pytest.mark.parametrize("dtype,tokens,hidden,intermediate,experts", [
    (torch.bfloat16, 256, 512, 256, 8),
    (torch.float16, 300, 256, 128, 4),
    (torch.bfloat16, 1024, 1024, 384, 16),
])
@pytest.mark.parametrize("block_size", [128, 256])
def test_moe_ffn_matches_oracle(cuda_device, dtype, tokens, hidden, intermediate, experts, block_size):
    data, ids, weights = _ffn_case(tokens, hidden, intermediate, experts, dtype, seed=11)
    ffn = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, block_size=block_size,
                      act_dtype="bf16" if dtype == torch.bfloat16 else "f16", target=ib.B200Target(0))
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    got_ids, got_weights = ffn.route(dev["logits"])
    assert torch.equal(got_ids.cpu(), ids)
    y = ffn(dev["x"], got_ids, got_weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"],
            dev["down_scales"])
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0
    ref = oracle.moe_w4a16_swiglu_ffn(data["x"], ids, weights, data["up_gate_packed"], data["up_gate_scales"],
                                      data["down_packed"], data["down_scales"])
    assert y.dtype == torch.float32 and y.shape == (tokens, hidden)
    assert max_abs_rel(y.cpu(), ref) <= 2e-2
    # deterministic: a second run gives the same bits
    y2 = ffn(dev["x"], got_ids, got_weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"],
             dev["down_scales"])
    assert torch.equal(y, y2)
    # bound once, replayed twice: same bits again
    y3 = torch.empty_like(y)
    call = ffn.prepare(dev["x"], got_ids, got_weights, dev["up_gate_packed"], dev["up_gate_scales"],
                       dev["down_packed"], dev["down_scales"], y3)
    call.launch()
    call.launch()
    assert torch.equal(y3, y)


def test_moe_ffn_benchmark_shape(cuda_device):
    """Benchmark configuration 4 at its own shape: 16384 tokens, H=4096, 64 experts, I=1408 (11 gate|up tiles
    per row block, down projection with K=1408 = 22 k blocks and 11 scale groups), top-2, bf16, g128, zp8,
    expert spans padded to 128.  A sample of tokens is compared with the oracle restricted to the experts
    those tokens use (tolerance 2e-2 * max|ref|, from the benchmark statement); run and prepared launch must
    give the same bits; a token-count checksum covers every token."""
    tokens, hidden, experts, inter = 16384, 4096, 64, 1408
    data = ib.workloads.moe_inputs(tokens, hidden, experts, inter, dtype=torch.bfloat16, seed=0)
    ids, weights = oracle.moe_route_top2(data["logits"])
    ffn = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=inter, experts=experts, block_size=128,
                      act_dtype="bf16", target=ib.B200Target(0))
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    got_ids, got_weights = ffn.route(dev["logits"])
    assert torch.equal(got_ids.cpu(), ids)
    args = (dev["x"], got_ids, got_weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"],
            dev["down_scales"])
    y = ffn(*args)
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0
    y2 = torch.full_like(y, float("nan"))
    call = ffn.prepare(*args, y2)
    call.launch()
    call.launch()
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0
    assert torch.equal(y, y2)
    assert torch.isfinite(y).all()

    # sample: first and last route (in the stable expert order) of the first, the two middle and the last
    # expert, tokens at both ends, and seeded random tokens: 72 tokens over most of the experts
    flat = ids.flatten().long()
    order = torch.argsort(flat, stable=True)
    counts = torch.bincount(flat, minlength=experts)
    starts = torch.cat((torch.zeros(1, dtype=torch.int64), counts.cumsum(0)))
    picked = []
    for expert in (0, 31, 32, 63):
        span = order[int(starts[expert]):int(starts[expert + 1])]
        picked += [int(span[0]) // 2, int(span[len(span) // 2]) // 2, int(span[-1]) // 2]
    picked += [0, 1, tokens - 2, tokens - 1]
    extra = torch.randperm(tokens, generator=torch.Generator().manual_seed(4))[:56].tolist()
    sample = torch.tensor(sorted(set(picked + extra)))
    assert sample.numel() >= 64
    # a token whose two experts live in different halves of the expert-sorted buffer (far-apart row blocks)
    assert any(abs(int(a) - int(b)) >= 32 for a, b in ids[sample].tolist())
    ref = oracle.moe_w4a16_swiglu_ffn(data["x"][sample], ids[sample], weights[sample], data["up_gate_packed"],
                                      data["up_gate_scales"], data["down_packed"], data["down_scales"])
    got = y[sample.to(cuda_device)].cpu()
    assert max_abs_rel(got, ref) <= 2e-2
    # per-token check as well: no sampled token may be far off on its own scale
    token_scale = ref.abs().amax(dim=1)
    assert ((got - ref).abs().amax(dim=1) <= 2e-2 * token_scale + 1e-6).all()


def test_grouped_entry_rejects_expert_ids_outside_the_table(cuda_device):
    """An expert id outside [0, E) in the block table must never be used as an index: the rows it governs
    are computed with zero weights and the status word reports INTENT_B200_ERR_INDEX (no fault)."""
    tokens, hidden, intermediate, experts = 256, 256, 128, 4
    data, ids, weights = _ffn_case(tokens, hidden, intermediate, experts, torch.bfloat16, seed=3)
    ffn = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    sorted_routes, expert_blocks, total = ffn.alignment.run(ids.to(cuda_device))
    rows = ffn.gather.run(dev["x"], sorted_routes, total)
    good = ffn.up_gate.run(rows, expert_blocks, total, dev["up_gate_packed"], dev["up_gate_scales"])
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0
    bad_blocks = expert_blocks.clone()
    bad_blocks[0] = experts + 3          # the first 128-row block names an expert that does not exist
    bad = ffn.up_gate.run(rows, bad_blocks, total, dev["up_gate_packed"], dev["up_gate_scales"])
    torch.cuda.synchronize()
    assert native.library().intent_b200_w4a16_gemm_device_status() == 8        # INTENT_B200_ERR_INDEX
    assert native.library().intent_b200_w4a16_gemm_device_status() == 0        # reading clears it
    assert not bad[:128].any()                                                  # zero weights -> zero rows
    first_good = 128 if int(expert_blocks[1]) != int(expert_blocks[0]) else 256
    assert torch.equal(bad[first_good:int(total)], good[first_good:int(total)])
    bad_blocks[0] = -1
    ffn.up_gate.run(rows, bad_blocks, total, dev["up_gate_packed"], dev["up_gate_scales"])
    with pytest.raises(ib.CompilationStageError):
        ffn.up_gate.check()


def test_grouped_projection_stage_by_stage(cuda_device):
    """The up|gate stage alone against the oracle's grouped product + SiLU gate."""
    tokens, hidden, intermediate, experts = 200, 256, 128, 4
    data, ids, weights = _ffn_case(tokens, hidden, intermediate, experts, torch.bfloat16, seed=2)
    ffn = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    sorted_routes, expert_blocks, total = ffn.alignment.run(ids.to(cuda_device))
    rows = ffn.gather.run(dev["x"], sorted_routes, total)
    hidden_act = ffn.up_gate.run(rows, expert_blocks, total, dev["up_gate_packed"], dev["up_gate_scales"])
    torch.cuda.synchronize()
    n = int(total)
    sorted_cpu = sorted_routes[:n].cpu().long()
    real = sorted_cpu < tokens * 2
    x_sorted = torch.zeros((n, hidden), dtype=torch.bfloat16)
    x_sorted[real] = data["x"][sorted_cpu[real] // 2]
    assert torch.equal(rows[:n].cpu(), x_sorted)
    expert_of_row = expert_blocks[: n // 128].cpu().long().repeat_interleave(128)
    gate_up = oracle.grouped_w4a16_gemm(x_sorted, expert_of_row, data["up_gate_packed"], data["up_gate_scales"],
                                        group_size=128, zero_point=8)
    ref = oracle.silu_and_mul(gate_up)
    assert max_abs_rel(hidden_act[:n].float().cpu(), ref) <= 2e-2


def test_host_pipelined_ffn_gives_the_whole_batch_bits(cuda_device):
    """Host tensors in and out, the batch cut into pieces that upload, run and download on three streams:
    tokens do not interact in this FFN, so the pieces give the bits the whole batch gives."""
    from intent_b200.moe import HostPipelinedFFN
    tokens, hidden, intermediate, experts = 512, 512, 256, 8
    data, ids, weights = _ffn_case(tokens, hidden, intermediate, experts, torch.bfloat16, seed=5)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    whole = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts,
                        target=ib.B200Target(0))
    got_ids, got_weights = whole.route(dev["logits"])
    expected = whole(dev["x"], got_ids, got_weights, dev["up_gate_packed"], dev["up_gate_scales"],
                     dev["down_packed"], dev["down_scales"]).cpu()
    piped = HostPipelinedFFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, chunks=4,
                             target=ib.B200Target(0)).bind(dev["up_gate_packed"], dev["up_gate_scales"],
                                                           dev["down_packed"], dev["down_scales"])
    logits, x = data["logits"].pin_memory(), data["x"].pin_memory()
    out = torch.empty((tokens, hidden), dtype=torch.float32).pin_memory()
    for _ in range(3):                       # buffers are reused from run to run
        out.zero_()
        piped.run(logits, x, out)
        assert torch.equal(out, expected)
    piped.check()
    with pytest.raises(ValueError):
        piped.run(logits[:100], x[:100], out[:100])
    with pytest.raises(ValueError):
        HostPipelinedFFN(tokens=510, hidden=hidden, intermediate=intermediate, experts=experts, chunks=4)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gate_over_its_range(cuda_device, dtype):
    """silu(g) * u against 64 bits for gates from the smallest to the largest, where the exponential is zero or infinite
    among them.  The result is rounded once (2^-11 of it in f16, 2^-8 in bf16) after f32 steps that are off by 2^-18 at most
    (__expf by 2 + 1.2 |g| units of 2^-24 with |g| up to 24, four roundings; beyond, the result is below 1e-6)."""
    ends = torch.tensor([0.0, 1e-6, 0.5, 16.0, 80.0, 87.0, 88.0, 88.5, 89.0, 104.0, 250.0])
    if dtype == torch.bfloat16:
        ends = torch.cat((ends, torch.tensor([1e4, 1e18])))
    spread = torch.randn((128 - 2 * ends.numel(),), generator=torch.Generator().manual_seed(1)) * 6
    values = torch.cat((ends, -ends, spread)).to(dtype)
    hidden, intermediate, experts = 128, 128, 1
    data = ib.workloads.moe_inputs(64, hidden, experts, intermediate, dtype=dtype, seed=1)
    x = torch.zeros((128, hidden), dtype=dtype)
    x[:, 0] = values                                                # times a weight of (9 - 8) * 1
    layer = MoEW4A16FFN(tokens=64, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0),
                        act_dtype="f16" if dtype == torch.float16 else "bf16")
    packed = torch.full_like(data["up_gate_packed"], int("99999999", 16) - 2 ** 32)
    out = layer.up_gate.run(x.to(cuda_device), torch.zeros(1, dtype=torch.int32, device=cuda_device),
                            torch.full((1,), 128, dtype=torch.int32, device=cuda_device), packed.to(cuda_device),
                            torch.ones_like(data["up_gate_scales"]).to(cuda_device)).cpu().double()
    g = values.double()
    exact = (g * torch.sigmoid(g) * g)[:, None].expand_as(out)
    largest = torch.finfo(dtype).max
    fits = exact.abs() < largest
    assert not torch.isnan(out).any() and torch.equal(out[~fits], exact[~fits].sign() * float("inf"))
    relative = (2 ** -11 if dtype == torch.float16 else 2 ** -8) + 2 ** -18
    assert ((out - exact).abs() <= relative * exact.abs() + 1e-6)[fits].all()


@pytest.mark.parametrize("prelayout", [False, True])
def test_a_layer_says_what_a_call_ran(cuda_device, prelayout):
    """``chain`` holds the programs of a call; ``gather`` and ``up_gate``, which take all rows, describe the call of the
    program that ran in their place until they are called themselves."""
    tokens, hidden, intermediate, experts = 64, 256, 128, 4
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=6)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0),
                        prelayout=prelayout)
    ids, weights = layer.route(dev["logits"])
    layer(dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    assert [p.observation.status for p in layer.chain] == [0, 0, 0]
    assert layer.chain[2] is layer.down_scatter
    for step, program in zip(layer.chain, (layer.gather, layer.up_gate)):
        seen, ran = program.observation, step.observation
        assert seen.status == 0 and (seen.entry, seen.arguments) == (ran.entry, ran.arguments)
    sorted_routes, _, total = layer.alignment.run(ids)
    layer.gather.run(dev["x"], sorted_routes, total)
    assert layer.gather.observation.entry == "intent_b200_moe_gather_rows"


def test_a_layer_says_what_the_latest_call_ran(cuda_device):
    """A call onto a ``y`` that is there, and a prepared one, run another up|gate program than a call that makes its own."""
    tokens, hidden, intermediate, experts = 64, 256, 128, 4
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=6)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    ids, weights = layer.route(dev["logits"])
    args = (dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    y = torch.zeros((tokens, hidden), dtype=torch.float32, device=cuda_device)
    for call, entry in ((lambda: layer(*args), "clear"), (lambda: layer(*args, y=y), "routed"), (lambda: layer(*args), "clear"),
                        (lambda: layer.prepare(*args, y).launch(), "routed")):
        call()
        assert layer.chain[1].observation.entry == f"intent_b200_moe_grouped_w4a16_upgate_silu_{entry}_bf16"
        assert layer.up_gate.observation.entry == layer.chain[1].observation.entry


@pytest.mark.parametrize("tokens,hidden", [(1, 128), (33, 1152), (300, 256)])
def test_a_call_clears_its_result(cuda_device, tokens, hidden):
    """The up|gate contraction zero-fills the result: whatever its memory held before, a call gives what adding to a zeroed
    ``y`` gives, bit for bit, and an unrouted token's row is zero."""
    intermediate, experts = 128, 4
    data, _, _ = _ffn_case(tokens, hidden, intermediate, experts, torch.bfloat16, seed=8)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    ids, weights = layer.route(dev["logits"])
    ids[-1] = -1                                                   # the last token goes nowhere
    args = (dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    expected = layer(*args, y=torch.zeros((tokens, hidden), dtype=torch.float32, device=cuda_device))
    for _ in range(4):
        stale = torch.full((tokens, hidden), float("nan"), dtype=torch.float32, device=cuda_device)
        del stale                                                  # (the result comes from this block)
        assert torch.equal(layer(*args), expected)
    assert not expected[-1].any()
    onto = torch.ones((tokens, hidden), dtype=torch.float32, device=cuda_device)
    assert layer(*args, y=onto) is onto and torch.equal(onto[-1], torch.ones_like(onto[-1]))
    with pytest.raises((TypeError, ValueError, RuntimeError)):     # one token more than there are weights
        layer(torch.cat((dev["x"], dev["x"][:1])), *args[1:])
    with pytest.raises(TypeError, match="route_weights must be a torch.Tensor"):
        layer(*args[:2], weights.tolist(), *args[3:])
    with pytest.raises(ValueError, match="rank"):
        layer(*args[:2], weights.sum(), *args[3:])


def test_a_call_clears_its_result_ahead(cuda_device):
    """Few tiles and a large result: it is filled ahead of the up|gate contraction, not beside it."""
    tokens, hidden, intermediate, experts = 1024, 4096, 128, 2
    data, ids, weights = _ffn_case(tokens, hidden, intermediate, experts, torch.bfloat16, seed=9)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, top_k=1,
                        target=ib.B200Target(0))
    args = (dev["x"], ids[:, :1].contiguous().to(cuda_device), weights[:, :1].contiguous().to(cuda_device),
            dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    expected = layer(*args, y=torch.zeros((tokens, hidden), dtype=torch.float32, device=cuda_device))
    for _ in range(4):
        stale = torch.full((tokens, hidden), float("nan"), dtype=torch.float32, device=cuda_device)
        del stale                                                  # (the result comes from this block)
        assert torch.equal(layer(*args), expected)
