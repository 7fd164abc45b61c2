"""Decode attention starts a large batch's longest requests first: a request's result does not depend on the batch around it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hkv,D,window", [(38, 8, 128, 0), (64, 8, 64, 0), (75, 4, 128, 100), (128, 8, 128, 0), (129, 8, 64, 0), (33, 16, 64, 0)])
def test_large_batches_match_small_ones(B, Hkv, D, window):
    from dinfer_b200.kernels import attention_ops
    H, page = 2 * Hkv, 16
    g = torch.Generator().manual_seed(B)
    lens = torch.randint(1, 700, (B,), generator=g, dtype=torch.int32)
    lens[1::5] = 300                                       # equal lengths
    new = torch.ones(B, dtype=torch.int32)
    new[::7] = 0                                           # places without a request
    new[3] = 5                                             # a portion: not this kernel's
    lens[::7], lens[3] = 0, 9
    cu = torch.cat([torch.zeros(1, dtype=torch.int32), new.cumsum(0).to(torch.int32)])
    most = 44
    table = torch.randperm(B * most, generator=g).to(torch.int32).view(B, most)
    cache = torch.randn(B * most, 2, Hkv, page, D, generator=g).to(torch.bfloat16).cuda()
    T = int(cu[-1])
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16).cuda()
    cu, lens, table = cu.cuda(), lens.cuda(), table.cuda()

    def run(a, z):
        out = torch.full((T, H * D), -7.0, dtype=torch.bfloat16, device="cuda")
        attention_ops.attention_decode(q, out, cache, table[a:z].contiguous(), cu[a:z + 1].contiguous(), lens[a:z].contiguous(), H, Hkv, D,
                                       D ** -0.5, window, 1)
        return out

    whole = run(0, B)
    for a in range(0, B, 16):
        z = min(B, a + 16)
        part, rows = run(a, z), slice(int(cu[a]), int(cu[z]))
        assert torch.equal(whole[rows], part[rows])
    assert bool((whole[int(cu[3]):int(cu[4])] == -7.0).all())
