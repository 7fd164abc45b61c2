"""Decode attention from the projection's rows against the q/k kernel and the decode attention one behind the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [  # B, H, Hkv, page, splits, window, keep, chunked, norm weights, table, history
    (1, 16, 8, 64, 8, 0, 0, False, "bf16", True, 1000),
    (3, 8, 8, 16, 1, 0, 0, False, "f32", True, 200),
    (8, 32, 4, 8, 4, 100, 3, False, None, True, 700),
    (5, 20, 4, 128, 16, 64, 0, True, "bf16", False, 1500),
    (2, 14, 2, 32, 3, 0, 0, False, None, False, 64),
    (40, 16, 8, 16, 1, 0, 0, False, "bf16", True, 300),      # more blocks than run at a time: the longest first
]


@pytest.mark.parametrize("case", CASES)
def test_raw_rows(case):
    from dinfer_b200.kernels import attention_ops, ops
    B, H, Hkv, page, splits, window, keep, chunked, weights, turned, history = case
    D, blocks = 128, -(-(history + 1) // page)
    g = torch.Generator().manual_seed(B + H)
    lens = torch.randint(1, history + 2, (B,), generator=g, dtype=torch.int32)
    lens[0] = history + 1
    if B > 2:
        lens[1], lens[2] = 1, page if page <= history else 2   # a token alone, a token that fills its page
    new = torch.ones(B, dtype=torch.int32)
    if B > 3:
        new[3] = 0                                            # a place without a request
    cu = torch.cat([torch.zeros(1, dtype=torch.int32), new.cumsum(0).to(torch.int32)])
    T = int(cu[-1])
    table = torch.randperm(B * blocks, generator=g).to(torch.int32).view(B, blocks)
    positions = torch.tensor([int(lens[b]) - 1 for b in range(B) if new[b]], dtype=torch.int32)
    rows = [b for b in range(B) if new[b]]
    slots = torch.tensor([int(table[b, (int(lens[b]) - 1) // page]) * page + (int(lens[b]) - 1) % page for b in rows], dtype=torch.int32)
    if T > 4:
        slots[4] = -1                                         # nowhere to put it
    cache = torch.randn(B * blocks, 2, Hkv, page, D, generator=g).to(torch.bfloat16).cuda()
    wide = (torch.randn(T, (H + 2 * Hkv) * D + 24, generator=g) * 2).to(torch.bfloat16).cuda()
    qkv = wide[:, :(H + 2 * Hkv) * D]
    w = [None, None]
    if weights:
        w = [(1 + 0.2 * torch.randn(D, generator=g)).to(torch.float32 if weights == "f32" else torch.bfloat16).cuda() for _ in range(2)]
    angles = torch.rand(history + 2, D // 2, generator=g) * 6.28
    cos_sin = torch.cat([angles.cos(), angles.sin()], 1).float().cuda() if turned else None
    c = lambda t: t.cuda()
    cu, lens, table, positions, slots = c(cu), c(lens), c(table), c(positions), c(slots)
    sinks = torch.randn(H, generator=g).cuda() if window else None
    slopes = (0.01 * torch.rand(H, generator=g)).cuda() if not turned else None
    seen = dict(chunked=chunked, keep_first=keep, sinks=sinks, slopes=slopes)

    got_cache, got, before = cache.clone(), torch.full((T, H * D), 7.0, dtype=torch.bfloat16, device="cuda"), wide.clone()
    attention_ops.attention_decode_raw(qkv, got, got_cache, table, cu, lens, H, Hkv, D ** -0.5, window, splits, positions, slots, 1e-6,
                                       w[0], w[1], cos_sin, **seen)
    assert torch.equal(wide, before)
    want_cache, want = cache.clone(), torch.full((T, H * D), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.qk_post(qkv, positions, H, Hkv, D, 1e-6, w[0], w[1], cos_sin, want_cache, slots, page)
    attention_ops.attention_decode(qkv[:, :H * D], want, want_cache, table, cu, lens, H, Hkv, D, D ** -0.5, window, splits, **seen)
    # the same arithmetic; a compiler may contract a product and a sum of one kernel and not of the other: an ulp of bfloat16
    # (2^-7 of a value) in a few places
    for a, b in ((got_cache, want_cache), (got, want)):
        a, b = a.float(), b.float()
        assert bool(((a - b).abs() <= b.abs() * 2 ** -7 + 2 ** -9).all()) and float((a != b).float().mean()) < 0.01


def test_what_it_does_not_take():
    from dinfer_b200.kernels import attention_ops as A
    x = torch.zeros(1, 1024, dtype=torch.bfloat16, device="cuda")
    assert A.decode_raw_supported(x, 128, 8, 8, 128, False, 0.0) and A.decode_raw_supported(x, 128, 1, 64, 0, False, 0.0)
    for args in ((x, 64, 1, 16, 64, False, 0.0), (x, 128, 9, 16, 128, False, 0.0), (x, 128, 2, 4, 128, False, 0.0),
                 (x, 128, 2, 16, 64, False, 0.0), (x, 128, 2, 16, 128, True, 0.0), (x, 128, 2, 16, 128, False, 30.0),
                 (x.float(), 128, 2, 16, 128, False, 0.0), (x[:, 1:], 128, 2, 16, 128, False, 0.0)):
        assert not A.decode_raw_supported(*args)
