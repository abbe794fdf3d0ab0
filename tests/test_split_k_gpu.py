"""Tiles whose k blocks are shared by a cluster: edges in rows, columns and k, the smallest and largest clusters, and calls that
ask for more tiles than they have clusters.  Which form a call runs on is read from its observation."""
import pytest
import torch

import intent_b200 as ib
import oracle

pytestmark = pytest.mark.gpu
TARGET = ib.B200Target(0)


@pytest.mark.parametrize("M,K,N,ctas", [
    (1, 6400, 16, 8),          # one row, sixteen columns: chunks that nobody owns
    (26, 5520, 4336, 4),       # 16 columns in the last tile, 16 k in the last block
    (96, 8192, 1040, 8),       # the most rows that eight CTAs share
    (97, 8192, 1040, 4),       # a fourth quadrant of one row
    (128, 4112, 4112, 4),      # 33 k blocks over four
    (200, 4096, 1024, 4),      # two row tiles, the second ragged
    (40, 2448, 16400, 2),      # twenty k blocks over two, 16 k in the last
])
@pytest.mark.parametrize("scaled", [False, True])
def test_int8(cuda_device, M, K, N, ctas, scaled):
    g = torch.Generator().manual_seed(M)
    a = torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-128, 128, (K, N), generator=g, dtype=torch.int8)
    if scaled:
        more = [torch.rand((n,), generator=g) * 0.01 + 1e-3 for n in (M, N)]
        expected = oracle.w8a8_scaled_gemm(a, b, *more)[0]
    else:
        more = [torch.randint(-2 ** 31, 2 ** 31, (N,), generator=g).to(torch.int32)]
        expected = oracle.gemm_i8_exact_f64(a, b, *more)
    artifact = ib.compile(ib.programs.w8a8_gemm if scaled else ib.programs.gemm_i8, target=TARGET)
    inputs = [t.to(cuda_device) for t in (a, b, *more)]
    for _ in range(3):
        out = artifact.run(*inputs)
    torch.cuda.synchronize()
    artifact.check()
    seen = artifact.observation
    assert seen.kernel.endswith("k split over a cluster") and seen.cluster == ctas, (seen.kernel, seen.cluster)
    assert torch.equal(out.cpu(), expected)


@pytest.mark.parametrize("dtype,rows,K,N", [
    (torch.bfloat16, (95, 32), 2392, 2104),              # K and N ragged
    (torch.float16, (0, 1, 0, 130, 3), 4096, 264),       # empty groups, two row blocks, eight columns in the last tile
    (torch.bfloat16, (64,), 8192, 520),
])
def test_ragged(cuda_device, dtype, rows, K, N):
    g = torch.Generator().manual_seed(K)
    x = torch.randn((sum(rows), K), generator=g).to(dtype)
    w = (torch.randn((len(rows), K, N), generator=g) * K ** -0.5).to(dtype)
    offsets = torch.tensor((0,) + rows).cumsum(0).to(torch.int32)
    program = ib.programs.ragged_grouped_gemm_bf16 if dtype == torch.bfloat16 else ib.programs.ragged_grouped_gemm
    artifact = ib.compile(program, target=TARGET)
    xd, od, wd = x.to(cuda_device), offsets.to(cuda_device), w.to(cuda_device)
    out = artifact.run(xd, od, wd)
    assert torch.equal(artifact.run(xd, od, wd), out)
    torch.cuda.synchronize()
    artifact.check()
    assert artifact.observation.kernel.endswith("k split over a cluster")
    exact = torch.cat([xd[a:b].double() @ wd[i].double() for i, (a, b) in enumerate(zip(offsets[:-1], offsets[1:]))])
    # f32 sums of 16-bit products and one rounding: half a unit in the last place of the value, or of the root mean square
    # where terms cancel (the sums' own error is below a hundredth of that)
    scale = exact.abs().clamp(min=exact.pow(2).mean().sqrt().item())
    assert ((out.double() - exact).abs() / scale).max() <= (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11) * 1.05


def test_offsets_that_do_not_rise(cuda_device):
    """Groups that overlap ask for more tiles than rows say: whole tiles then, and every row is written."""
    rows, K, N = 300, 2048, 512
    g = torch.Generator().manual_seed(1)
    x = torch.randn((rows, K), generator=g).to(torch.bfloat16).to(cuda_device)
    one = (torch.randn((1, K, N), generator=g) * K ** -0.5).to(torch.bfloat16)
    w = one.expand(9, K, N).contiguous().to(cuda_device)          # the same weights, so that it does not matter who writes
    offsets = torch.tensor([0, rows] * 5, dtype=torch.int32, device=cuda_device)
    artifact = ib.compile(ib.programs.ragged_grouped_gemm_bf16, target=TARGET)
    out = artifact.run(x, offsets, w)
    torch.cuda.synchronize()
    artifact.check()
    exact = x.double() @ one[0].to(cuda_device).double()
    scale = exact.abs().clamp(min=exact.pow(2).mean().sqrt().item())
    assert ((out.double() - exact).abs() / scale).max() <= 2 ** -8 * 1.05


def test_expert_ffn(cuda_device):
    """The weighted add of a tile that a cluster shares: once per element, by its owner."""
    tokens, D, F, experts = 40, 2048, 2048, 2
    g = torch.Generator().manual_seed(2)
    x = torch.randn((tokens, D), generator=g).to(torch.float16)
    w1 = (torch.randn((experts, D, F), generator=g) * D ** -0.5).to(torch.float16)
    w2 = (torch.randn((experts, F, D), generator=g) * F ** -0.5).to(torch.float16)
    expert = torch.randint(0, experts, (tokens,), generator=g)
    members = torch.argsort(expert, stable=True).to(torch.int32)
    offsets = torch.zeros(experts + 1, dtype=torch.int32)
    offsets[1:] = torch.bincount(expert, minlength=experts).cumsum(0)
    token, weight = torch.arange(tokens, dtype=torch.int32), torch.rand((tokens,), generator=g)
    artifact = ib.compile(ib.programs.moe_expert_ffn, target=TARGET, constexprs={"DTYPE": "f16"})
    y = torch.zeros((tokens, D), dtype=torch.float32, device=cuda_device)
    artifact(*(t.to(cuda_device) for t in (x, offsets, members, token, weight, w1, w2)), y)
    torch.cuda.synchronize()
    artifact.check()
    hidden = torch.stack([torch.relu(x[t].double() @ w1[expert[t]].double()) for t in range(tokens)])
    exact = torch.stack([weight[t].double() * (hidden[t] @ w2[expert[t]].double()) for t in range(tokens)])
    # the hidden rows are rounded to f16 (2^-11 each) before F products are added: 2^-11 of the root mean square, and the
    # spread of 81920 values
    assert (y.cpu().double() - exact).abs().max() / exact.pow(2).mean().sqrt() <= 2 ** -11 * 6
