"""The routed feed-forward's layout, gather and small row tiles at the sizes where their passes change."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,pairs,tile,shift", [(1, 5, 16, 0), (64, 16384, 256, 0), (64, 4095, 64, 0), (33, 4096, 16, 1),
                                                (340, 8192, 16, 0), (341, 8190, 64, 0), (359, 8192, 16, 0), (360, 8190, 64, 0),
                                                (4095, 9000, 16, 0), (7, 0, 16, 0)])
def test_align_deals_every_pair_once(E, pairs, tile, shift):
    """Pairs of ids outside [0, E) are left out; every expert's run holds its pairs, then padding; nothing else is written."""
    from dinfer_b200.kernels import moe_ops
    ids = torch.randint(-1, E + 1, (pairs + shift,), dtype=torch.int32, device="cuda")[shift:]      # shift: no 16-byte loads
    if pairs:
        ids[: pairs // 2] = E // 2                                                                  # one crowded expert
    sorted_, tile_expert = moe_ops.align(ids, E, tile)
    ids, sorted_, tile_expert = ids.tolist(), sorted_.tolist(), tile_expert.tolist()
    want = {}
    for i, e in enumerate(ids):
        if 0 <= e < E:
            want.setdefault(e, set()).add(i)
    row = 0
    for e in sorted(want):
        n = -(-len(want[e]) // tile) * tile
        assert set(sorted_[row:row + len(want[e])]) == want[e]
        assert sorted_[row + len(want[e]):row + n] == [pairs] * (n - len(want[e]))
        assert tile_expert[row // tile:(row + n) // tile] == [e] * (n // tile)
        row += n
    assert set(sorted_[row:]) <= {pairs} and set(tile_expert[row // tile:]) <= {-1}


@pytest.mark.parametrize("h,dtype,top,shift", [(8, torch.bfloat16, 1, 0), (2048, torch.bfloat16, 4, 0), (2056, torch.bfloat16, 2, 0),
                                               (4104, torch.bfloat16, 2, 0), (264, torch.bfloat16, 2, 4), (37, torch.bfloat16, 3, 0),
                                               (100, torch.float32, 2, 0)])
def test_gather_rows(h, dtype, top, shift):
    from dinfer_b200.kernels import moe_ops
    T, E = 61, 9
    x = torch.randn(T, h + shift, device="cuda").to(dtype)[:, shift:]                               # shift: rows off 16 bytes
    ids = torch.randint(0, E, (T * top,), dtype=torch.int32, device="cuda")
    sorted_, _ = moe_ops.align(ids, E, 16)
    a = moe_ops.gather_rows(x, sorted_, T * top, top)
    real = sorted_ < T * top
    assert torch.equal(a[real], x[(sorted_[real] // top).long()])


@pytest.mark.parametrize("K", [8, 56, 64, 72, 192, 200, 256, 264, 2048])
@pytest.mark.parametrize("N", [64, 72])
def test_small_row_tiles(K, N):
    """Both products on row tiles of 16: K below, at and beyond the four stages of 64, a ragged last column tile."""
    from dinfer_b200.kernels import moe_ops
    T, top, E = 11, 2, 5
    g = torch.Generator().manual_seed(K + N)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    ids = torch.randint(0, E, (T * top,), generator=g, dtype=torch.int32).cuda()
    p = torch.rand(T * top, generator=g).cuda()
    sorted_, tile_expert = moe_ops.align(ids, E, 16)
    real = sorted_ < T * top
    pair = sorted_[real].long()
    want = torch.einsum("pk,pnk->pn", x.float()[pair // top], w.float()[ids[pair].long()])
    out = torch.empty(sorted_.numel(), N, dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm(x, w, out, sorted_, tile_expert, T * top, top, 16, 0)
    # one rounding to bfloat16 (2^-8 of the value at most) and sums of K products in 32 bits
    assert bool(((out[real].float() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all())
    a = torch.zeros(sorted_.numel(), K, dtype=torch.bfloat16, device="cuda")
    a[real] = x[pair // top]
    y = torch.full((T * top, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm(a, w, y, sorted_, tile_expert, T * top, top, 16, 1, weights=p)
    want = want * p[pair, None]
    assert bool(((y[pair].float() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all())


@pytest.mark.parametrize("N", [40, 1000, 1280, 2440, 4800])
@pytest.mark.parametrize("K", [136, 384])
def test_small_row_tiles_dealt(N, K):
    """Runs of 0 to 17 rows an expert (one tile or two, one half of a tile or both) and products of less than a round of the
    device's CTAs, dealt whole, in halves and in quarters, or of a round and a rest; a row's bits are its own, whatever is
    beside it."""
    from dinfer_b200.kernels import moe_ops
    counts = [1, 8, 9, 16, 17, 0, 2, 3]
    E, T = len(counts), sum(counts)
    g = torch.Generator().manual_seed(K + N)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=g)].int().cuda()
    want = torch.einsum("pk,pnk->pn", x.float(), w.float()[ids.long()])
    got = []
    for keep in (torch.arange(T), torch.arange(T)[::5]):                   # all rows, and some of them alone
        xs, es = x[keep].contiguous(), ids[keep.cuda()].contiguous()
        sorted_, tile_expert = moe_ops.align(es, E, 16)
        out = torch.empty(sorted_.numel(), N, dtype=torch.bfloat16, device="cuda")
        moe_ops.grouped_gemm(xs, w, out, sorted_, tile_expert, len(keep), 1, 16, 0)
        real = sorted_ < len(keep)
        y = torch.empty(len(keep), N, dtype=torch.bfloat16, device="cuda")
        y[sorted_[real].long()] = out[real]
        # one rounding to bfloat16 (2^-8 of the value at most) and sums of K products in 32 bits
        assert bool(((y.float() - want[keep.cuda()]).abs() <= want[keep.cuda()].abs() * 2 ** -8 + 1e-4).all())
        got.append(y)
    assert torch.equal(got[1], got[0][::5])


@pytest.mark.parametrize("gate", ["silu", "gelu_tanh", "relu", "relu2", ("clamped_swish", 7.0, 1.702)])
@pytest.mark.parametrize("N", [32, 74, 320])
def test_small_row_tiles_gate(gate, N):
    """The gate in the first product against the product's bfloat16 results gated in 32 bits."""
    from dinfer_b200.kernels import moe_ops
    T, K, E = 37, 200, 3
    g = torch.Generator().manual_seed(N)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, N, K, generator=g) * 3 * K ** -0.5).to(torch.bfloat16).cuda()
    ids = torch.randint(0, E, (T,), generator=g, dtype=torch.int32).cuda()
    sorted_, tile_expert = moe_ops.align(ids, E, 16)
    real = sorted_ < T
    plain = torch.empty(sorted_.numel(), N, dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm(x, w, plain, sorted_, tile_expert, T, 1, 16, 0)
    out = torch.empty(sorted_.numel(), N // 2, dtype=torch.bfloat16, device="cuda")
    moe_ops.grouped_gemm(x, w, out, sorted_, tile_expert, T, 1, 16, 0, gate=gate)
    a, u = plain[real][:, 0::2].float(), plain[real][:, 1::2].float()
    if isinstance(gate, tuple):
        a, u = a.clamp(max=7.0), u.clamp(-7.0, 7.0)
        want = a * torch.sigmoid(1.702 * a) * (u + 1)
    else:
        want = u * {"silu": lambda z: z * torch.sigmoid(z), "relu": torch.relu, "relu2": lambda z: torch.relu(z) ** 2,
                    "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh")}[gate](a)
    # one rounding to bfloat16, 2^-8 at most; the 32-bit gates differ by a few 2^-22 of values below 100
    assert bool(((out[real].float() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all())
    with pytest.raises(moe_ops.KernelError):
        moe_ops.grouped_gemm(x, w, out, sorted_, tile_expert, T, 1, 16, 1, gate=gate)
    with pytest.raises(moe_ops.KernelError):
        moe_ops.grouped_gemm(x[:, 1:], w[:, :, 1:].contiguous(), out, sorted_, tile_expert, T, 1, 16, 0, gate=gate)
