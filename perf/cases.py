"""Performance cases: the calls a user of this framework makes, over the sizes it is used at.

Every case goes through the public surface - ``intent_b200.compile(...).run``, ``W4A16Table`` and
``MoEW4A16FFN`` - with inputs drawn on the GPU from the seed.  ``listed()`` holds the fixed cases, ``draw``
gives further ones of the same ranges, ``prepare`` makes what a program has in hand before the call (inputs,
weights and the compiled artifact or bound call it keeps), ``run`` is one pass.
"""
from __future__ import annotations

import math

import torch

import intent_b200 as ib
from intent_b200.moe import MoEW4A16FFN
from intent_b200.table import W4A16Table

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # One token of a decode step through one projection (hidden 4096 -> intermediate 14336): a single
        # artifact call whose cost is the weight stream plus the launch and the call itself.
        {"name": "decode_gemv", "kind": "w4a16", "M": 1, "K": 4096, "N": 14336, "dtype": "f16", "group": 128,
         "zero": 8},
        # The two projections of a decode step bound once into one table and launched per token.
        {"name": "decode_table", "kind": "table", "M": 1, "hidden": 4096, "intermediate": 14336, "dtype": "f16",
         "group": 128, "zero": 8},
        # A decode step of sixteen sequences on a square projection.
        {"name": "decode_rows16", "kind": "w4a16", "M": 16, "K": 4096, "N": 4096, "dtype": "f16", "group": 128,
         "zero": 8},
        # A short prompt or a large decode batch: an odd row count between the decode and the prefill sizes, on
        # the down projection (long K).
        {"name": "rows77_down", "kind": "w4a16", "M": 77, "K": 14336, "N": 4096, "dtype": "bf16", "group": 128,
         "zero": 8},
        # The program with its own default constants (group 64, two's complement nibbles, f16) at the size its
        # tests use.
        {"name": "rows512_group64", "kind": "w4a16", "M": 512, "K": 2048, "N": 4096, "dtype": "f16", "group": 64,
         "zero": "twos_complement"},
        # A long prefill: the largest dense contraction.
        {"name": "prefill_8192", "kind": "w4a16", "M": 8192, "K": 8192, "N": 8192, "dtype": "bf16", "group": 128,
         "zero": 8},
        # Int8 activations and weights with per-token and per-channel scales, prefill size.
        {"name": "w8a8_prefill", "kind": "i8", "M": 4096, "K": 8192, "N": 8192, "scaled": True},
        # A mixture-of-experts layer over a prefill batch: router, alignment, both expert projections, combine.
        {"name": "moe_prefill", "kind": "moe", "tokens": 16384, "hidden": 4096, "intermediate": 1408, "experts": 64,
         "dtype": "bf16"},
        # The same layer for a decode batch: every expert sees a few rows, so the experts' weights are the cost.
        {"name": "moe_decode", "kind": "moe", "tokens": 64, "hidden": 4096, "intermediate": 1408, "experts": 64,
         "dtype": "bf16"},
        # Dense ragged contraction over groups of unequal size.
        {"name": "ragged_bf16", "kind": "ragged", "rows": "256-512-1024-2048", "K": 4096, "N": 4096, "dtype": "bf16"},
        # Dense 16-bit expert FFN over routed rows, the largest of the dense programs.
        {"name": "expert_ffn_f16", "kind": "expert_ffn", "tokens": 4096, "D": 4096, "F": 14336, "experts": 8,
         "dtype": "f16"},
        # One row against two-bit weights: the smallest call, where the launch and the call itself count.
        {"name": "int2_decode", "kind": "packed", "program": "bitnet_int2_matmul", "M": 1, "K": 4096, "N": 4096},
    ]


def _size(rng, low, high, multiple):
    """A size between ``low`` and ``high``, even over its logarithm, a multiple of ``multiple``."""
    return max(multiple, int(round(math.exp(rng.uniform(math.log(low), math.log(high))) / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["w4a16", "w4a16", "w4a16", "table", "i8", "moe", "moe", "ragged", "expert_ffn", "packed"])
    dtype = rng.choice(["f16", "bf16"])
    if kind in ("w4a16", "table"):
        group = rng.choice([32, 64, 128, 128])
        zero = rng.choice([8, "twos_complement"])
        if kind == "table":
            return {"kind": kind, "M": rng.randint(1, 8), "hidden": _size(rng, 1024, 8192, 128),
                    "intermediate": _size(rng, 2048, 14336, 128), "dtype": dtype, "group": group, "zero": zero}
        return {"kind": kind, "M": _size(rng, 1, 8192, 1), "K": _size(rng, 1024, 8192, group),
                "N": _size(rng, 1024, 8192, 8), "dtype": dtype, "group": group, "zero": zero}
    if kind == "i8":
        return {"kind": kind, "M": _size(rng, 16, 4096, 1), "K": _size(rng, 1024, 8192, 16),
                "N": _size(rng, 1024, 8192, 16), "scaled": rng.random() < 0.5}
    if kind == "moe":
        return {"kind": kind, "tokens": _size(rng, 1, 16384, 1), "hidden": _size(rng, 1024, 4096, 128),
                "intermediate": _size(rng, 512, 1408, 128), "experts": rng.choice([8, 16, 32, 64]), "dtype": dtype}
    if kind == "ragged":
        rows = [_size(rng, 16, 2048, 1) for _ in range(rng.randint(2, 8))]
        return {"kind": kind, "rows": "-".join(map(str, rows)), "K": _size(rng, 1024, 4096, 8),
                "N": _size(rng, 1024, 4096, 8), "dtype": dtype}
    if kind == "expert_ffn":
        return {"kind": kind, "tokens": _size(rng, 64, 4096, 1), "D": _size(rng, 1024, 4096, 8),
                "F": _size(rng, 2048, 14336, 8), "experts": 8, "dtype": dtype}
    program = rng.choice(["bitnet_int2_matmul", "w4a8_packed_matmul", "dequant_bf16_fp4_matmul",
                          "quantized_projection"])
    K, N = _size(rng, 1024, 8192, 256), _size(rng, 1024, 8192, 16)
    M = {"bitnet_int2_matmul": _size(rng, 1, 1024, 1), "w4a8_packed_matmul": _size(rng, 16, 4096, 16),
         "dequant_bf16_fp4_matmul": _size(rng, 1, 4096, 1), "quantized_projection": 1}[program]
    return {"kind": kind, "program": program, "M": M, "K": K, "N": N}


# ---- inputs ---------------------------------------------------------------------------------------------------
class _Source:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.generator = torch.Generator(device=self.device).manual_seed(int(seed))

    def normal(self, shape, dtype, scale=1.0):
        if math.prod(shape) > 1 << 28:   # large weights are drawn plane by plane
            return torch.stack([self.normal(shape[1:], dtype, scale) for _ in range(shape[0])])
        return (torch.randn(shape, generator=self.generator, device=self.device) * scale).to(dtype)

    def integers(self, low, high, shape, dtype):
        return torch.randint(low, high, shape, generator=self.generator, device=self.device, dtype=dtype)

    def words(self, shape):
        """Packed int4 weights: every nibble uniform."""
        return self.integers(-2 ** 31, 2 ** 31, shape, torch.int64).to(torch.int32)

    def scales(self, shape, dtype):
        return (0.002 + 0.01 * torch.randn(shape, generator=self.generator, device=self.device).abs()).to(dtype)

    def permutation(self, count):
        return torch.randperm(count, generator=self.generator, device=self.device)


def _w4a16(source, M, K, N, dtype, group):
    return (source.normal((M, K), dtype), source.words((K // 8, N)), source.scales((K // group, N), dtype))


def _fp16_bytes(values):
    return values.to(torch.float16).unsqueeze(-1).view(torch.uint8)


def prepare(case, seed):
    source, kind = _Source(seed), case["kind"]
    target = ib.B200Target(torch.cuda.current_device())
    dtype = DTYPES.get(case.get("dtype"))
    if kind == "w4a16":
        artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=target, constexprs={
            "GROUP_SIZE": case["group"], "ZERO_POINT": case["zero"], "ACT_DTYPE": case["dtype"]})
        return {"kind": kind, "call": artifact.run,
                "inputs": _w4a16(source, case["M"], case["K"], case["N"], dtype, case["group"])}
    if kind == "table":
        table = W4A16Table(group_size=case["group"], zero_point=case["zero"], act_dtype=case["dtype"], target=target)
        shapes = [(case["hidden"], case["intermediate"]), (case["intermediate"], case["hidden"])]
        return {"kind": kind, "call": table.prepare([_w4a16(source, case["M"], K, N, dtype, case["group"])
                                                     for K, N in shapes])}
    if kind == "i8":
        M, K, N = case["M"], case["K"], case["N"]
        a = source.integers(-127, 128, (M, K), torch.int8)
        b = source.integers(-127, 128, (K, N), torch.int8)
        if case["scaled"]:
            scale = [0.01 * source.normal((n,), torch.float32).abs() + 1e-3 for n in (M, N)]
            return {"kind": kind, "call": ib.compile(ib.programs.w8a8_gemm, target=target).run,
                    "inputs": (a, b, *scale)}
        return {"kind": kind, "call": ib.compile(ib.programs.gemm_i8, target=target).run,
                "inputs": (a, b, source.integers(-1000, 1000, (N,), torch.int32))}
    if kind == "moe":
        T, H, I, E = case["tokens"], case["hidden"], case["intermediate"], case["experts"]
        layer = MoEW4A16FFN(tokens=T, hidden=H, intermediate=I, experts=E, act_dtype=case["dtype"], target=target)
        weights = (source.words((E, H // 8, 2 * I)), source.scales((E, H // 128, 2 * I), dtype),
                   source.words((E, I // 8, H)), source.scales((E, I // 128, H), dtype))
        return {"kind": kind, "layer": layer, "logits": source.normal((T, E), torch.float32),
                "x": source.normal((T, H), dtype, H ** -0.5), "weights": weights}
    if kind == "ragged":
        rows = [int(r) for r in case["rows"].split("-")]
        K, N = case["K"], case["N"]
        offsets = torch.tensor([0] + rows, device=source.device).cumsum(0).to(torch.int32)
        program = ib.programs.ragged_grouped_gemm_bf16 if case["dtype"] == "bf16" else ib.programs.ragged_grouped_gemm
        return {"kind": kind, "call": ib.compile(program, target=target).run,
                "inputs": (source.normal((sum(rows), K), dtype), offsets,
                           source.normal((len(rows), K, N), dtype, K ** -0.5))}
    if kind == "expert_ffn":
        T, D, F, E = case["tokens"], case["D"], case["F"], case["experts"]
        # two choices per token; routes listed expert by expert
        first = source.integers(0, E, (T,), torch.int64)
        second = (first + 1 + source.integers(0, E - 1, (T,), torch.int64)) % E
        expert = torch.stack([first, second], 1).reshape(-1)
        members = torch.argsort(expert, stable=True).to(torch.int32)
        offsets = torch.zeros((E + 1,), dtype=torch.int32, device=source.device)
        offsets[1:] = torch.bincount(expert, minlength=E).cumsum(0).to(torch.int32)
        token = torch.arange(T, device=source.device, dtype=torch.int32).repeat_interleave(2)
        share = torch.rand((T, 2), generator=source.generator, device=source.device) + 0.1
        weights = (share / share.sum(1, keepdim=True)).reshape(-1).contiguous()
        artifact = ib.compile(ib.programs.moe_expert_ffn, target=target, constexprs={"DTYPE": case["dtype"]})
        return {"kind": kind, "call": artifact.run, "shape": (T, D), "device": source.device,
                "inputs": (source.normal((T, D), dtype), offsets, members, token, weights,
                           source.normal((E, D, F), dtype, D ** -0.5), source.normal((E, F, D), dtype, F ** -0.5))}
    program, M, K, N = case["program"], case["M"], case["K"], case["N"]
    call = ib.compile(getattr(ib.programs, program), target=target).run
    if program == "quantized_projection":
        records = source.integers(0, 256, (N, K // 256, 144), torch.uint8)
        for at, size in ((0, 0.01), (2, 0.005)):     # the record's two half-precision factors
            factor = size * torch.rand((N, K // 256), generator=source.generator, device=source.device)
            records[:, :, at:at + 2] = _fp16_bytes(factor)
        inputs = (records, source.normal((K // 256, 256), torch.float32))
    elif program == "dequant_bf16_fp4_matmul":
        inputs = (source.normal((M, K), torch.bfloat16), source.integers(0, 256, (N, K // 2), torch.uint8))
    else:
        per_byte = 4 if program == "bitnet_int2_matmul" else 2
        inputs = (source.integers(-127, 128, (M, K), torch.int8),
                  source.integers(0, 256, (N, K // per_byte), torch.uint8))
    return {"kind": kind, "call": call, "inputs": inputs}


def run(state):
    kind = state["kind"]
    if kind == "table":
        state["call"].launch()
        return state["call"].results()
    if kind == "moe":
        ids, weights = state["layer"].route(state["logits"])
        return ids, weights, state["layer"](state["x"], ids, weights, *state["weights"])
    if kind == "expert_ffn":
        y = torch.zeros(state["shape"], dtype=torch.float32, device=state["device"])
        state["call"](*state["inputs"], y)
        return y
    return state["call"](*state["inputs"])


def work(case):
    kind = case["kind"]

    def w4a16(M, K, N, group):
        return K * N / 2 + 2 * (K // group) * N + 2 * M * K + 2 * M * N, 2 * M * K * N

    if kind == "w4a16":
        size, flops = w4a16(case["M"], case["K"], case["N"], case["group"])
    elif kind == "table":
        parts = [w4a16(case["M"], K, N, case["group"]) for K, N in ((case["hidden"], case["intermediate"]),
                                                                   (case["intermediate"], case["hidden"]))]
        size, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "i8":
        M, K, N = case["M"], case["K"], case["N"]
        size = M * K + K * N + (2 * M * N + 4 * M if case["scaled"] else 4 * M * N) + 4 * N
        flops = 2 * M * K * N
    elif kind == "moe":
        T, H, I, E = case["tokens"], case["hidden"], case["intermediate"], case["experts"]
        used = E * (1 - (1 - 2 / E) ** T)              # experts with at least one of the 2 T routes
        size = used * 3 * H * I * (0.5 + 2 / 128) + 6 * T * H + 4 * T * E + 16 * T
        flops = 2 * T * 2 * 3 * H * I
    elif kind == "ragged":
        rows = [int(r) for r in case["rows"].split("-")]
        K, N = case["K"], case["N"]
        size = 2 * (sum(rows) * (K + N) + len(rows) * K * N)
        flops = 2 * sum(rows) * K * N
    elif kind == "expert_ffn":
        T, D, F, E = case["tokens"], case["D"], case["F"], case["experts"]
        size = 4 * E * D * F + 2 * T * D + 4 * T * D + 24 * T
        flops = 2 * T * 2 * 2 * D * F
    else:
        M, K, N = case["M"], case["K"], case["N"]
        act, weight, out = {"bitnet_int2_matmul": (1, 0.25, 4), "w4a8_packed_matmul": (1, 0.5, 4),
                            "dequant_bf16_fp4_matmul": (2, 0.5, 2),
                            "quantized_projection": (4, 144 / 256, 4)}[case["program"]]
        size, flops = M * K * act + K * N * weight + M * N * out, 2 * M * K * N
    return {"bytes": float(size), "flops": float(flops)}


def tolerance(case):
    kind = case["kind"]
    if kind == "i8":
        # the s32 accumulator is exact; the scaled form rounds once to bf16
        return {"rel": 1e-3} if case["scaled"] else "exact"
    if kind == "packed":
        if case["program"] == "quantized_projection":
            return {"rel": 1e-5}
        return {"rel": 8e-3} if case["program"] == "dequant_bf16_fp4_matmul" else "exact"
    # 16-bit operands and results with f32 sums; the int4 weight may be rounded to the activation type before the
    # product and the expert FFN's hidden rows are.  Against the same formulas in 64 bits the kernels differ by
    # 1.7e-3 .. 3.0e-3 in bf16 and 2.1e-4 .. 3.8e-4 in f16 (2-norms): four times the largest of each.
    return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1.5e-3}
