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
