"""The W4A16 kernel with the weights in tensor memory: edges of its tiles in rows, columns and k.  Tiled weight copies
run on the other kernels, which add the k blocks in the same order, so unsplit calls must agree with them bit for bit;
the tolerances against the oracle are those of test_w4a16_gemm_gpu.py."""
import threading

import pytest
import torch

import intent_b200 as ib
import oracle
from intent_b200 import prelayout
from intent_b200.moe import MoEW4A16FFN
from intent_b200.runtime import native
from conftest import max_abs_rel

pytestmark = pytest.mark.gpu

LONE, PAIRS, SPLIT = ("w4a16_tmem_kernel " + s for s in ("single CTA", "CTA pairs", "k split over a cluster"))


@pytest.mark.parametrize("dtype,zero_point,group,M,K,N,kernel", [
    (torch.float16, 8, 128, 17, 4096, 4096, SPLIT),                    # one tile of 32 rows, four CTAs a tile
    (torch.bfloat16, "twos_complement", 32, 77, 4128, 2056, SPLIT),    # a quarter of a k block at the end, 33 blocks
    (torch.bfloat16, 8, 64, 130, 2112, 9224, LONE),                    # half a k block, a ragged second row tile
    (torch.float16, "twos_complement", 64, 512, 2048, 4096, LONE),
    (torch.bfloat16, 8, 128, 511, 8192, 8200, PAIRS),                  # 256-row tiles, one accumulator
    (torch.float16, 8, 128, 1030, 4096, 4104, PAIRS),                  # 128-row tiles, eight columns in the last tile
    (torch.bfloat16, 8, 128, 35, 2048, 19208, LONE),                   # more tiles than SMs, three rows past a chunk of 32
    (torch.float16, 8, 128, 33, 8192, 1032, SPLIT),                    # eight CTAs a tile
    (torch.float16, "twos_complement", 32, 36, 1184, 1000, LONE),      # the shortest K, a quarter of a block at its end
    (torch.bfloat16, 8, 128, 546, 1408, 1112, LONE),                   # twelve row tiles of 48
    (torch.bfloat16, 8, 64, 2180, 2112, 1224, PAIRS),                  # more than 2047 rows
])
def test_dense_tiles(cuda_device, dtype, zero_point, group, M, K, N, kernel):
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=dtype, group_size=group, seed=M)
    constants = {"GROUP_SIZE": group, "ZERO_POINT": zero_point, "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"}
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0), constexprs=constants)
    tiled = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                       constexprs=dict(constants, WEIGHT_LAYOUT="tiled", KERNEL="gemm"))
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    out = artifact.run(xd, pd, sd)
    assert artifact.observation.kernel.startswith(kernel), artifact.observation.kernel
    assert torch.equal(artifact.run(xd, pd, sd), out)
    other = tiled.run(xd, prelayout.tile(pd).tensor, sd)
    torch.cuda.synchronize()
    artifact.check()
    if kernel is not SPLIT:
        assert torch.equal(out, other)
    rows = torch.randperm(M, generator=torch.Generator().manual_seed(1))[:128].sort().values
    rows = torch.cat([torch.tensor([0]), rows, torch.tensor([M - 1])])
    rounded = oracle.weight_only_int4_matmul_rounded(x[rows], p, s, group_size=group,
                                                     zero_point=8 if zero_point == 8 else None)
    assert max_abs_rel(out[rows.to(cuda_device)].cpu(), rounded) <= (2e-3 if dtype == torch.float16 else 1.6e-2)


@pytest.mark.parametrize("dtype,zero_point,group,M,K,N", [
    (torch.float16, 8, 128, 16, 4096, 4096),                     # four CTAs a tile
    (torch.bfloat16, "twos_complement", 32, 9, 1056, 136),       # four groups a k block, a quarter block at the end
    (torch.float16, "twos_complement", 64, 13, 2112, 1000),
    (torch.bfloat16, 8, 128, 12, 2048, 19208),                   # more tiles than SMs
    (torch.bfloat16, 8, 64, 13, 8256, 520),                      # eight CTAs a tile, four of which own no row
    (torch.float16, 8, 128, 5, 4096, 9472),                      # the fewest rows, on the most columns that they may have
    (torch.bfloat16, "twos_complement", 32, 8, 1056, 1032),
    (torch.bfloat16, 8, 64, 7, 2112, 9608),                      # more tiles than half the SMs
])
def test_nine_to_sixteen_rows(cuda_device, dtype, zero_point, group, M, K, N):
    """Scales in f32, as in the bandwidth kernels: no further from the result in 64 bits than they are."""
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=dtype, group_size=group, seed=M)
    constants = {"GROUP_SIZE": group, "ZERO_POINT": zero_point, "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"}
    artifact, other = (ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                                  constexprs=dict(constants, KERNEL=kernel)) for kernel in ("auto", "gemv"))
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    out, stream = artifact.run(xd, pd, sd), other.run(xd, pd, sd)
    assert artifact.observation.kernel.startswith("w4a16_tmem_kernel 16 rows"), artifact.observation.kernel
    assert torch.equal(artifact.run(xd, pd, sd), out)
    torch.cuda.synchronize()
    artifact.check()
    q = oracle.unpack_int4(p).double()
    q = q - 8 if zero_point == 8 else torch.where(q > 7, q - 16, q)
    exact = x.double() @ (q * s.double().repeat_interleave(group, dim=0))
    error, before = ((o.cpu().double() - exact).norm() / exact.norm() for o in (out, stream))
    assert error <= before * 1.02       # both are the rounding of the result; 2 % for sums in another order


@pytest.mark.parametrize("dtype,group,M,K,N,kernel", [
    (torch.float16, 128, 7, 14592, 5144, "w4a16_ride_kernel"),      # 57 k blocks for each of 82 CTAs
    (torch.bfloat16, 32, 8, 6656, 13448, "w4a16_ride_kernel"),      # tiles that cannot be cut
    (torch.bfloat16, 64, 5, 10496, 160, "w4a16_tmem_kernel 16 rows"),
    (torch.float16, 128, 8, 2048, 13448, "w4a16_tmem_kernel 16 rows"),
    (torch.float16, 128, 4, 4096, 4096, "w4a16_ride_kernel"),
])
def test_four_to_eight_rows(cuda_device, dtype, group, M, K, N, kernel):
    """On either side of the line between the two kernels the result is as far from 64 bits as the bandwidth kernel's."""
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=dtype, group_size=group, seed=M)
    constants = {"GROUP_SIZE": group, "ZERO_POINT": 8, "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"}
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0), constexprs=constants)
    out = artifact.run(x.to(cuda_device), p.to(cuda_device), s.to(cuda_device))
    assert artifact.observation.kernel.startswith(kernel), artifact.observation.kernel
    torch.cuda.synchronize()
    artifact.check()
    exact = x.double() @ ((oracle.unpack_int4(p).double() - 8) * s.double().repeat_interleave(group, dim=0))
    rounded = exact.to(dtype).double()
    assert (out.cpu().double() - exact).norm() <= 1.02 * (rounded - exact).norm()   # the rounding of the result; 2 % for the sums


@pytest.mark.parametrize("rows_of_expert,hidden,intermediate,block", [
    ((1, 16, 17, 0, 32, 33, 15, 2), 512, 128, 128),            # few rows: lone CTAs
    ((127, 128, 129, 0, 256, 1, 300, 31), 1024, 384, 128),     # blocks full and nearly empty: CTA pairs
    ((127, 128, 129, 0, 256, 1, 300, 31), 256, 128, 256),      # blocks of 256 rows, the second half empty
])
def test_routed_rows(cuda_device, rows_of_expert, hidden, intermediate, block):
    experts = len(rows_of_expert)
    flat = torch.repeat_interleave(torch.arange(experts), torch.tensor(rows_of_expert))
    flat = flat[torch.randperm(flat.numel(), generator=torch.Generator().manual_seed(2))]
    ids = flat[: flat.numel() // 2 * 2].reshape(-1, 2).to(torch.int32)
    tokens = ids.shape[0]
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=3)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    weights = torch.rand((tokens, 2), generator=torch.Generator().manual_seed(4))
    sizes = dict(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, block_size=block,
                 target=ib.B200Target(0))
    args = (dev["x"], ids.to(cuda_device), weights.to(cuda_device), dev["up_gate_packed"], dev["up_gate_scales"],
            dev["down_packed"], dev["down_scales"])
    plain, tiled = MoEW4A16FFN(**sizes), MoEW4A16FFN(prelayout=True, **sizes)
    y = plain(*args)
    assert plain.chain[1].observation.kernel.startswith("w4a16_tmem_kernel")
    torch.cuda.synchronize()
    plain.down_scatter.check()
    assert torch.equal(y, tiled(*args))
    ref = oracle.moe_w4a16_swiglu_ffn(data["x"], ids, weights, data["up_gate_packed"], data["up_gate_scales"],
                                      data["down_packed"], data["down_scales"])
    assert max_abs_rel(y.cpu(), ref) <= 2e-2


@pytest.mark.parametrize("M,K,N,group", [(8, 1056, 1032, 32), (13, 2112, 520, 64), (300, 2048, 2056, 128)])
def test_scales_at_the_end_of_the_range(cuda_device, M, K, N, group):
    """bfloat16 scales up to 2^124 beside ordinary ones: times the weight they are finite, and so is the result.  An
    infinite or NaN scale reaches its own column only."""
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=torch.bfloat16, group_size=group, seed=M)
    x = (x.float() * 2.0 ** -40).to(torch.bfloat16)
    picked = torch.rand(s.shape, generator=torch.Generator().manual_seed(1)) < 0.02
    exponents = torch.randint(118, 125, s.shape, generator=torch.Generator().manual_seed(2))
    s = torch.where(picked, 2.0 ** exponents.float(), s.float()).to(torch.bfloat16)
    s[:, 7] = 2.0 ** 124
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": group, "ZERO_POINT": 8, "ACT_DTYPE": "bf16"})
    xd, pd = x.to(cuda_device), p.to(cuda_device)
    out = artifact.run(xd, pd, s.to(cuda_device))
    assert artifact.observation.kernel.startswith("w4a16_tmem_kernel"), artifact.observation.kernel
    exact = x.double() @ ((oracle.unpack_int4(p).double() - 8) * s.double().repeat_interleave(group, dim=0))
    assert torch.isfinite(out).all()
    # (a sum's terms are rounded to 2^-9 of their size and so is the result, and terms are no larger than eight times x times s)
    worst = x.double().abs() @ (8 * s.double().repeat_interleave(group, dim=0))
    assert ((out.cpu().double() - exact).abs() <= 2 ** -8 * worst).all()
    s[0, 3], s[1, 5] = float("inf"), float("nan")
    broken = artifact.run(xd, pd, s.to(cuda_device))
    good = torch.ones(N, dtype=torch.bool)
    good[[3, 5]] = False
    assert torch.equal(broken[:, good], out[:, good]) and not torch.isfinite(broken[:, ~good]).any()


def test_grouped_scales_at_the_end_of_the_range(cuda_device):
    tokens, hidden, intermediate, experts = 300, 512, 256, 4
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=6)
    data["down_scales"][:, 0, ::3] = 2.0 ** 123
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    sizes = dict(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    plain, tiled = MoEW4A16FFN(**sizes), MoEW4A16FFN(prelayout=True, **sizes)
    ids, weights = plain.route(dev["logits"])
    # hidden rows small enough for sums of 2^126 times them to stay finite
    args = ((dev["x"].float() * 2.0 ** -12).to(torch.bfloat16), ids, weights, dev["up_gate_packed"], dev["up_gate_scales"],
            dev["down_packed"], dev["down_scales"])
    y = plain(*args)
    assert torch.isfinite(y).all() and torch.equal(y, tiled(*args))


@pytest.mark.parametrize("tokens,hidden,intermediate", [
    (1024, 4096, 128), (5120, 4096, 128),     # one k block in the down projection; 3.5 and 17.3 tiles a CTA or pair
    (1024, 4096, 256), (5120, 4096, 256),
    (1024, 4096, 384), (2048, 4096, 384),     # three; 3.5 and 6.9
    (1024, 128, 2048), (1280, 128, 8192),     # the same for up|gate
    (1024, 256, 2048), (1280, 256, 8192),
    (1024, 384, 2048),
])
def test_several_tiles_of_few_k_blocks(cuda_device, tokens, hidden, intermediate):
    """The dequantiser warps take rows of a CTA's last tile: only once it is complete, also where all of a set's blocks are
    out before the tiles ahead have been multiplied."""
    experts = 8                               # full blocks of 128 rows: every expert has tokens / 4 of them
    first = torch.arange(tokens) % experts
    ids = torch.stack([first, (first + 3) % experts], 1).to(torch.int32)
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=tokens + hidden)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    weights = torch.rand((tokens, 2), generator=torch.Generator().manual_seed(4)) + 0.1
    sizes = dict(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    args = (dev["x"], ids.to(cuda_device), weights.to(cuda_device), dev["up_gate_packed"], dev["up_gate_scales"],
            dev["down_packed"], dev["down_scales"])
    rows_args = args[:2] + args[3:]
    plain, tiled = MoEW4A16FFN(**sizes), MoEW4A16FFN(prelayout=True, **sizes)
    expected, rows = tiled(*args), tiled.experts_forward(*rows_args)[0]      # (no block has padding rows)
    library = native.library()
    try:
        for pairs in (1, 0):
            library.intent_b200_w4a16_gemm_pairs(pairs)
            for _ in range(8):
                y = plain(*args)
                assert plain.down_scatter.observation.kernel.startswith(PAIRS if pairs else LONE)
                assert torch.equal(y, expected)
                assert torch.equal(plain.experts_forward(*rows_args)[0][:2 * tokens], rows[:2 * tokens])
    finally:
        library.intent_b200_w4a16_gemm_pairs(1)
    torch.cuda.synchronize()
    plain.down_scatter.check()
    some = torch.arange(0, tokens, tokens // 64)
    ref = oracle.moe_w4a16_swiglu_ffn(data["x"][some], ids[some], weights[some], data["up_gate_packed"],
                                      data["up_gate_scales"], data["down_packed"], data["down_scales"])
    assert max_abs_rel(expected[some.to(cuda_device)].cpu(), ref) <= 2e-2


@pytest.mark.parametrize("sizes", [
    ((32, 2176, 512), (128, 2176, 512)),     # one instance of this kernel, 214528 and 224768 bytes of shared memory
    ((1, 1024, 512), (1, 4096, 4096)),       # the bandwidth kernel: rings of a few slots and of many
    ((4, 1024, 512), (4, 4096, 4096)),       # a table of one problem
])
def test_threads_launch_one_instance(cuda_device, sizes):
    """Calls of one kernel instance with different shared memory do not get in each other's way: a launch must not fail
    because another thread has asked for less in between."""
    failures, threads = [], []

    def work(M, K, N):
        x, p, s = (t.to(cuda_device) for t in ib.workloads.w4a16_inputs(M, K, N, dtype=torch.bfloat16, seed=M))
        artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                              constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8, "ACT_DTYPE": "bf16"})
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                expected = artifact.run(x, p, s)
                ready.wait(60)
                for _ in range(40):
                    for _ in range(100):
                        out = artifact.run(x, p, s)
                    torch.cuda.current_stream().synchronize()      # (a full queue would keep the threads apart)
            if not torch.equal(out, expected):
                failures.append((M, "other bits"))
        except Exception as error:
            failures.append((M, str(error)))
            ready.abort()

    ready = threading.Barrier(4 * len(sizes))
    torch.cuda.synchronize()
    for size in 4 * sizes:
        threads.append(threading.Thread(target=work, args=size))
        threads[-1].start()
    for t in threads:
        t.join()
    assert not failures, failures[:1]


@pytest.mark.parametrize("dtype,group,K,N", [
    (torch.bfloat16, 128, 4096, 4096),
    (torch.float16, 64, 2112, 2056),         # half a k block at the end, eight columns in the last tile
])
def test_rows_of_one_kernel_keep_their_bits(cuda_device, dtype, group, K, N):
    """KERNEL='gemm' adds the k blocks in one order whatever else a call holds: the bits of a row depend neither on the
    number of rows, nor on the columns beside it, nor on the layout of the weights.  The default may cut K into two, four
    or eight parts for few rows; the same products are then added in f32 in another order, so that results agree to the rounding
    of the output type (half a unit in the last place each: 2^-8 of the value in bf16, 2^-11 in f16; cancellation leaves
    sums that are small against their terms, hence the root mean square beside the value)."""
    M = 2100                                 # runs on another kernel
    x, p, s = ib.workloads.w4a16_inputs(M, K, N, dtype=dtype, group_size=group, seed=K)
    constants = {"GROUP_SIZE": group, "ZERO_POINT": 8, "ACT_DTYPE": "f16" if dtype == torch.float16 else "bf16"}
    compiled = lambda **more: ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                                         constexprs=dict(constants, **more))
    auto, gemm, tiled = compiled(), compiled(KERNEL="gemm"), compiled(KERNEL="gemm", WEIGHT_LAYOUT="tiled")
    xd, pd, sd = x.to(cuda_device), p.to(cuda_device), s.to(cuda_device)
    whole = gemm.run(xd, pd, sd)
    assert not gemm.observation.kernel.startswith("w4a16_tmem_kernel")
    assert torch.equal(tiled.run(xd, prelayout.tile(pd).tensor, sd), whole)
    half = slice(0, N // 16 * 8)
    shard = pd[:, half].contiguous(), sd[:, half].contiguous()
    split = 0
    for rows in (1, 17, 32, 77, 128, 200, 511, 1300):
        part = xd[:rows].contiguous()
        assert torch.equal(gemm.run(part, pd, sd), whole[:rows]), rows
        assert "split" not in gemm.observation.kernel
        assert torch.equal(gemm.run(part, *shard), whole[:rows, half]), rows
        if rows > 16:
            out = auto.run(part, pd, sd).double()
            split += "split" in auto.observation.kernel
            scale = whole[:rows].double().abs().clamp(min=whole.double().pow(2).mean().sqrt().item())
            assert ((out - whole[:rows].double()).abs() / scale).max() <= (2 ** -10 if dtype == torch.float16 else 2 ** -7)
    assert split
    torch.cuda.synchronize()
    gemm.check()


def test_the_pairs_switch_holds_for_grouped_calls(cuda_device):
    """With pairs switched off the grouped contractions run on lone CTAs, with the same bits."""
    library = native.library()
    tokens, hidden, intermediate, experts = 1024, 512, 256, 4
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=5)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    layer = MoEW4A16FFN(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    ids, weights = layer.route(dev["logits"])
    args = (dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    paired = layer(*args)
    assert layer.down_scatter.observation.kernel.startswith(PAIRS)
    try:
        assert library.intent_b200_w4a16_gemm_pairs(0) == 0
        single = layer(*args)
        assert layer.down_scatter.observation.kernel.startswith(LONE)
    finally:
        library.intent_b200_w4a16_gemm_pairs(1)
    assert torch.equal(single, paired)


def test_more_row_blocks_than_the_kernel_lists(cuda_device):
    """Above 1024 blocks of 128 rows a grouped call runs on the kernel with the weights in shared memory, here with a row
    or none for each of many experts; the rows of padding hold whatever was there before."""
    tokens, hidden, intermediate, experts = 96, 384, 128, 1040
    data = ib.workloads.moe_inputs(tokens, hidden, experts, intermediate, dtype=torch.bfloat16, seed=7)
    dev = {k: v.to(cuda_device) for k, v in data.items()}
    sizes = dict(tokens=tokens, hidden=hidden, intermediate=intermediate, experts=experts, target=ib.B200Target(0))
    plain, tiled = MoEW4A16FFN(**sizes), MoEW4A16FFN(prelayout=True, **sizes)
    ids, weights = plain.route(dev["logits"])
    args = (dev["x"], ids, weights, dev["up_gate_packed"], dev["up_gate_scales"], dev["down_packed"], dev["down_scales"])
    stale = torch.full((1 << 26,), float("nan"), dtype=torch.bfloat16, device=cuda_device)
    del stale                                    # the rows and the hidden rows of the call come from this block
    y = plain(*args)
    assert plain.down_scatter.observation.kernel.startswith("w4a16_gemm_kernel")
    assert torch.equal(y, tiled(*args))
    torch.cuda.synchronize()
    plain.down_scatter.check()
    ref = oracle.moe_w4a16_swiglu_ffn(data["x"], ids.cpu(), weights.cpu(), data["up_gate_packed"], data["up_gate_scales"],
                                      data["down_packed"], data["down_scales"])
    assert max_abs_rel(y.cpu(), ref) <= 2e-2


def test_dependent_calls_without_synchronisation(cuda_device):
    """Programmatic launches: a call starts while the one before it is still running, and must see what that one wrote -
    activations from another kernel of this library, and weights that were copied just before.  Twelve rows, four, one and
    77 by turns; the same chain with a synchronisation after every step gives the expected bits."""
    width, steps = 2176, 48
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8, "ACT_DTYPE": "bf16"})
    x, p, s = ib.workloads.w4a16_inputs(77, width, width, dtype=torch.bfloat16, seed=8)
    others = [ib.workloads.w4a16_inputs(1, width, width, dtype=torch.bfloat16, seed=9 + i)[1].to(cuda_device) for i in (0, 1)]
    xd, sd = x.to(cuda_device), s.to(cuda_device)
    kernels = set()

    def chain(synchronise):
        weight, state = others[0].clone(), xd.clone()
        for step in range(steps):
            rows = (12, 4, 1, 77)[step % 4]
            weight.copy_(others[step % 2])
            out = artifact.run(state[:rows], weight, sd)
            if synchronise:
                torch.cuda.synchronize()
                kernels.add(artifact.observation.kernel.split(",")[0])
            state = torch.cat((out, state[rows:]))
            if rows == 77:       # and one call straight after another
                state = artifact.run(artifact.run(state[:16], weight, sd), weight, sd).repeat(5, 1)[:77]
            state = state / state.abs().amax(dim=1, keepdim=True)
        return state

    expected = chain(True)
    assert torch.isfinite(expected).all() and len(kernels) == 4, kernels
    for _ in range(10):
        assert torch.equal(chain(False), expected)
