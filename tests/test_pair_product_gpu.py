"""The two-SM product at every width its token tiles can have, dense and grouped by experts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want):
    # one rounding to bfloat16 (2^-8 of the value at most) and sums of some hundred products of order 0.1 in 32 bits
    return bool(((got.float() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all())


@pytest.mark.parametrize("tokens", [65, 96, 128, 129, 192, 193, 255, 256, 257, 320, 449, 777])
@pytest.mark.parametrize("N,K", [(256, 64), (130, 136), (777, 200), (600, 72)])
def test_dense(tokens, N, K):
    from dinfer_b200.kernels import gemm_ops
    g = torch.Generator().manual_seed(tokens + N)
    x = torch.randn(tokens, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    want = x.float() @ w.float().t()
    for dtype in (torch.bfloat16, torch.float32):
        wide = torch.full((tokens + 1, N + 3), 7.0, dtype=dtype, device="cuda")
        out = wide[:tokens, :N]                               # rows that no 4-byte or 8-byte pair of columns fits evenly
        gemm_ops.gemm_tc(x, w, out)
        assert close(out, want) and bool((wide[tokens:] == 7.0).all()) and bool((wide[:, N:] == 7.0).all())
        flat = torch.empty(tokens, N, dtype=dtype, device="cuda")
        assert torch.equal(gemm_ops.gemm_tc(x, w, flat), out)
    if N % 2 == 0:
        act = torch.empty(tokens, N // 2, dtype=torch.bfloat16, device="cuda")
        gemm_ops.gemm_tc(x, w, act, gated=True)
        assert close(act, torch.nn.functional.silu(want[:, ::2]) * want[:, 1::2])


RUNS = [[256] * 3, [1, 0, 31, 32, 33, 63, 64, 65], [0, 127, 128, 129, 191, 193, 255, 257, 300, 511, 512, 513, 0]]


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("N,K", [(256, 72), (264, 136), (520, 64)])
def test_grouped(runs, N, K):
    from dinfer_b200.kernels import moe_ops
    E, pairs = len(runs), sum(runs)
    g = torch.Generator().manual_seed(pairs + N)
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(runs)])[torch.randperm(pairs, generator=g)].cuda()
    x = torch.randn(pairs, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    p = torch.rand(pairs, generator=g).cuda()
    sorted_, tile_expert = moe_ops.align(ids, E, moe_ops.TC_ROW_TILE)
    real = sorted_ < pairs
    at = sorted_[real].long()
    want = torch.stack([x[i].float() @ w[ids[i].item()].float().t() for i in range(pairs)])
    a = torch.full((sorted_.numel(), K), float("nan"), dtype=torch.bfloat16, device="cuda")      # rows that pad hold anything
    a[real] = x[at]
    out = torch.empty(sorted_.numel(), N, dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm_tc(a, w, out, sorted_, tile_expert, pairs, 0)
    assert close(out[real], want[at])
    moe_ops.grouped_gemm_tc(a, w, out, sorted_, tile_expert, pairs, 0, activation="silu")
    assert close(out[real], torch.nn.functional.silu(want[at]))
    half = torch.empty(sorted_.numel(), N // 2, dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm_tc(a, w, half, sorted_, tile_expert, pairs, 0, gate="silu")
    assert close(half[real], (torch.nn.functional.silu(want[:, ::2]) * want[:, 1::2])[at])
    y = torch.full((pairs, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm_tc(a, w, y, sorted_, tile_expert, pairs, 1, weights=p)
    assert close(y, want * p[:, None])
