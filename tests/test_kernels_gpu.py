"""Each kernel alone against a plain torch reference of the same operation, at sizes other than the
engine's tiny models (widths and vocabularies that are no power of two, head sizes in steps of 16,
odd head and group counts)."""
import math
import random

import pytest
import torch

import plain_model as P

pytestmark = pytest.mark.gpu

DT = [torch.float32, torch.bfloat16]


def tol(dt):
    return dict(atol=2e-5, rtol=2e-5) if dt == torch.float32 else dict(atol=2e-2, rtol=2e-2)


def dev(t, dt=None):
    return t.to("cuda", dtype=dt) if dt else t.to("cuda")


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("T,h", [(1, 24), (7, 1000), (33, 4100), (3, 20000)])
def test_rmsnorm_add_and_gather(dt, T, h):
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(T * h)
    res = torch.randn(T, h, generator=g) * 3
    delta = (torch.randn(T, h, generator=g)).to(dt)
    w = (1 + 0.3 * torch.randn(h, generator=g)).to(dt)
    eps = 1e-5
    # plain norm of the residual
    r = dev(res.clone())
    out = torch.empty(T, h, dtype=dt, device="cuda")
    ops.rmsnorm(r, dev(w), eps, out)
    want = P.rms_norm(res.double(), w.double(), eps)
    assert torch.allclose(out.double().cpu(), want, **tol(dt))
    assert torch.equal(r.cpu(), res)
    # fused add: residual updated in place, in 32-bit
    ops.rmsnorm(r, dev(w), eps, out, delta=dev(delta))
    summed = res + delta.float()
    assert torch.equal(r.cpu(), summed)
    assert torch.allclose(out.double().cpu(), P.rms_norm(summed.double(), w.double(), eps), **tol(dt))
    # gather of rows (+ pending delta), residual untouched
    rows = torch.tensor([T - 1, 0, T // 2], dtype=torch.int32)
    r2 = dev(res.clone())
    out2 = torch.empty(3, h, dtype=dt, device="cuda")
    ops.rmsnorm(r2, dev(w), eps, out2, delta=dev(delta), rows=dev(rows))
    assert torch.equal(r2.cpu(), res)
    assert torch.allclose(out2.double().cpu(), P.rms_norm(summed.double(), w.double(), eps)[rows.long()], **tol(dt))


@pytest.mark.parametrize("dt", DT)
def test_embedding_and_silu(dt):
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(5)
    table = torch.randn(301, 72, generator=g).to(dt)
    ids = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32)
    out = torch.empty(5, 72, dtype=torch.float32, device="cuda")
    ops.embedding(dev(ids), dev(table), out)
    assert torch.equal(out.cpu(), table.float()[ids.long()])
    ops.embedding(dev(ids), dev(table), out, scale=8.48528137)    # a model that scales its embedding
    assert torch.allclose(out.cpu(), table.float()[ids.long()] * 8.48528137, rtol=1e-6, atol=0)
    logits = (torch.randn(3, 1001, generator=g) * 40).float()    # a soft cap on logits, in place
    capped = ops.softcap(dev(logits).clone(), 30.0)
    assert torch.allclose(capped.cpu().double(), 30.0 * torch.tanh(logits.double() / 30.0), rtol=1e-5, atol=1e-5)
    x = (torch.randn(9, 2 * 250, generator=g) * 4).to(dt)
    o = torch.empty(9, 250, dtype=dt, device="cuda")
    ops.silu_mul(dev(x), o)
    xd = x.double()
    want = P.silu(xd[:, :250]) * xd[:, 250:]
    assert torch.allclose(o.double().cpu(), want, **tol(dt))
    for inter in (250, 256, 44):                              # gate and up side by side, vector and plain paths
        x = (torch.randn(7, 2 * inter, generator=g) * 4).to(dt)
        o = torch.empty(7, inter, dtype=dt, device="cuda")
        ops.silu_mul(dev(x), o, pairs=True)
        xd = x.double()
        assert torch.allclose(o.double().cpu(), P.silu(xd[:, 0::2]) * xd[:, 1::2], **tol(dt))


@pytest.mark.parametrize("M,N,K", [(1, 37, 50), (8, 130, 999), (9, 260, 70), (130, 129, 1031), (300, 17, 8)])
@pytest.mark.parametrize("adt,wdt,cdt", [(torch.float32,) * 3, (torch.bfloat16, torch.float32, torch.bfloat16),
                                         (torch.float32, torch.bfloat16, torch.float32)])
def test_gemm_f32(M, N, K, adt, wdt, cdt):
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(M * N + K)
    a = torch.randn(M, K, generator=g).to(adt)
    w = torch.randn(N, K, generator=g).to(wdt)
    out = torch.empty(M, N, dtype=cdt, device="cuda")
    ops.gemm_f32(dev(a), dev(w), out)
    want = a.double() @ w.double().T
    t = dict(atol=1e-4 * math.sqrt(K), rtol=1e-5) if cdt == torch.float32 else dict(atol=5e-2 * math.sqrt(K) / 8, rtol=1e-2)
    assert torch.allclose(out.double().cpu(), want, **t)


@pytest.mark.parametrize("M,N,K", [(9, 129, 16), (64, 128, 132), (65, 127, 260), (128, 256, 1024), (333, 1024, 3072), (64, 8, 2050),
                                   (40, 20, 4), (9, 48, 48), (25, 5, 129), (32, 2049, 128), (31, 2048, 128), (17, 33, 1)])
@pytest.mark.parametrize("adt,wdt,cdt", [(torch.float32,) * 3, (torch.bfloat16, torch.float32, torch.bfloat16),
                                         (torch.float32, torch.bfloat16, torch.float32)])
def test_gemm_f32_tiles_and_splits(M, N, K, adt, wdt, cdt):
    """Edges of the tile, remainders of a stage, one to eight CTAs to a tile's K, aligned rows and rows that are not.  K
    products summed in any order in 32-bit are off by at most (K + 1) 2^-24 of the sum of their sizes, plus the rounding of
    a bfloat16 result (2^-8 of it)."""
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N + K)
    for pad in (0, 1):                                       # rows of whole 16-byte pieces, and rows that are not
        a = torch.randn(M, K + pad, generator=g).to(adt)[:, :K]
        w = torch.randn(N, K + pad, generator=g).to(wdt)[:, :K]
        out = torch.full((M, N + pad), float("nan"), dtype=cdt, device="cuda")
        da, dw = dev(torch.cat([a, a[:, :pad]], 1))[:, :K], dev(torch.cat([w, w[:, :pad]], 1))[:, :K]
        ops.gemm_f32(da, dw, out[:, :N])
        want = a.double() @ w.double().T
        bound = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
        if cdt == torch.bfloat16:
            bound = bound + 2.0 ** -8 * want.abs()
        assert bool(((out[:, :N].double().cpu() - want).abs() <= bound).all())
        assert pad == 0 or bool(torch.isnan(out[:, N:]).all())
    # several problems at once, their rows interleaved
    a = torch.randn(M, 3, 44, generator=g).to(adt)
    w = torch.randn(3, N, 44, generator=g).to(wdt)
    out = torch.full((M, 3, N), float("nan"), dtype=cdt, device="cuda")
    ops.gemm_f32_batched(dev(a), dev(w), out)
    want = torch.einsum("mbk,bnk->mbn", a.double(), w.double())
    bound = 45 * 2.0 ** -24 * torch.einsum("mbk,bnk->mbn", a.double().abs(), w.double().abs())
    if cdt == torch.bfloat16:
        bound = bound + 2.0 ** -8 * want.abs()
    assert bool(((out.double().cpu() - want).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(112, 128, 32), (113, 129, 33), (111, 127, 31), (224, 136, 68), (1, 200, 64), (33, 8, 4096), (256, 2048, 96)])
@pytest.mark.parametrize("batch", [1, 3])
def test_gemm_f32_extreme_values(M, N, K, batch):
    """Infinities, values that are not numbers and the largest ones give what plain 32-bit sums give; rows of tiny values keep
    their digits down to 2^-133 (what a split element keeps), rows with large and small values side by side theirs."""
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, batch, K, generator=g), torch.randn(batch, N, K, generator=g)
    a *= torch.exp(torch.randn(M, batch, 1, generator=g) * 6)            # rows of all sizes
    a[M // 2] *= torch.exp(torch.randn(batch, K, generator=g) * 4)
    a[M // 3] *= 2.0 ** -100
    plain = torch.einsum("mbk,bnk->mbn", a.double(), w.double())
    size = torch.einsum("mbk,bnk->mbn", a.double().abs(), w.double().abs())
    weight = w.double().abs().sum(2)                                      # [batch, N]
    bound = (K + 1) * 2.0 ** -24 * size + 2.0 ** -133 * weight[None]
    out = torch.full((M, batch, N), 7.0, device="cuda")
    ops.gemm_f32_batched(dev(a), dev(w), out)
    assert bool(((out.double().cpu() - plain).abs() <= bound).all())
    # one element of a row, one of a weight row: everything they do not meet is as before, bit for bit
    row, col, k = M - 1, N // 2, K - 1
    for bad in (math.inf, -math.inf, math.nan, 3.4028234e38):
        b = a.clone()
        b[row, batch - 1, k] = bad
        v = w.clone()
        v[0, col, k] = -bad
        got = torch.full((M, batch, N), 7.0, device="cuda")
        ops.gemm_f32_batched(dev(b), dev(v), got)
        want = torch.einsum("mbk,bnk->mbn", b.double(), v.double())
        rest = torch.ones(M, batch, N, dtype=torch.bool)
        rest[row, batch - 1] = False
        rest[:, 0, col] = False
        assert torch.equal(got.cpu()[rest], out.cpu()[rest])
        hit, want = got.cpu()[~rest], want[~rest]
        if math.isinf(bad) or math.isnan(bad):
            assert torch.equal(torch.isnan(hit), torch.isnan(want)) and torch.equal(hit[torch.isinf(hit)].double(), want[torch.isinf(hit)])
            assert bool((torch.isfinite(hit) == torch.isfinite(want)).all())
        else:                                                             # beyond 32-bit: infinite; else one large product
            big = want.abs() > 3.5e38
            assert bool((torch.isinf(hit[big])).all()) and torch.equal(torch.sign(hit[big]).double(), torch.sign(want[big]))
            fine = want.abs() < 3.3e38
            assert bool(((hit.double() - want).abs()[fine] <= (K + 1) * 2.0 ** -24 * 4 * 3.4028234e38).all())


@pytest.mark.parametrize("M", [65535 * 64, 65535 * 64 + 1, 65535 * 128])
def test_gemm_f32_of_millions_of_rows(M):
    """As many row tiles as a grid has, one more, and the most rows a product may have; one more is refused."""
    from dinfer_b200.kernels import ops
    from dinfer_b200.kernels.lib import KernelError
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn(M, 4, generator=g, device="cuda"), torch.randn(5, 4, generator=g, device="cuda")
    out = torch.full((M + 1, 5), 7.0, device="cuda")
    ops.gemm_f32(a, w, out[:M])
    # four products of a few units and their sum in 32-bit: 5 roundings of 2^-24
    assert float((out[:M].double() - a.double() @ w.double().T).abs().max()) <= 5 * 2.0 ** -24 * float(a.abs().max() * w.abs().max()) * 4
    assert bool((out[M] == 7.0).all())
    if M == 65535 * 128:
        with pytest.raises(KernelError, match="too large"):
            ops.gemm_f32(torch.zeros(M + 1, 1, device="cuda"), w[:, :1].contiguous(), torch.empty(M + 1, 5, device="cuda"))


def test_gemm_f32_strided_operands():
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    big = dev(torch.randn(20, 100, generator=g))
    a = big[:, 10:60]                       # row stride 100, 50 columns
    w = dev(torch.randn(31, 50, generator=g))
    outbig = torch.zeros(20, 64, device="cuda")
    ops.gemm_f32(a, w, outbig[:, 3:34])
    assert torch.allclose(outbig[:, 3:34], a @ w.T, atol=1e-4)
    assert float(outbig[:, :3].abs().max()) == 0 and float(outbig[:, 34:].abs().max()) == 0


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H,Hkv,D,rot,bs", [(4, 1, 16, 16, 4), (6, 2, 32, 32, 16), (5, 5, 48, 48, 8),
                                             (8, 2, 128, 64, 16), (3, 3, 256, 256, 32), (2, 1, 80, 80, 16),
                                             (32, 8, 128, 128, 16), (5, 1, 128, 128, 16), (16, 8, 128, 128, 8),
                                             (6, 2, 64, 64, 16)])
def test_qk_post(dt, H, Hkv, D, rot, bs):
    from dinfer_b200.kernels import ops
    from dinfer_b200.parts.rope import rope_table
    g = torch.Generator().manual_seed(H * D)
    T, nb, eps, theta, maxpos = 11, 9, 1e-5, 12345.0, 300
    width = (H + 2 * Hkv) * D
    qkv = torch.randn(T, width + 8, generator=g).to(dt)           # padded rows: stride != width
    pos = torch.tensor(random.Random(1).sample(range(maxpos), T), dtype=torch.int32)
    wq = (1 + 0.2 * torch.randn(D, generator=g)).to(dt)
    wk = (1 + 0.2 * torch.randn(D, generator=g)).to(dt)
    slots = torch.tensor(random.Random(2).sample(range(nb * bs), T), dtype=torch.int32)
    slots[3] = -1
    cache = torch.zeros(nb, 2, Hkv, bs, D, dtype=dt, device="cuda")
    table = rope_table(rot, theta, maxpos, "cuda")
    x = dev(qkv)
    ops.qk_post(x[:, :width], dev(pos), H, Hkv, D, eps, dev(wq), dev(wk), table, cache, dev(slots), bs)
    # plain
    q = qkv[:, :H * D].double().reshape(T, H, D)
    k = qkv[:, H * D:(H + Hkv) * D].double().reshape(T, Hkv, D)
    v = qkv[:, (H + Hkv) * D:width].double().reshape(T, Hkv, D)
    cos, sin = P.rope_cos_sin(pos, rot, theta)
    qn, kn = P.rms_norm(q, wq.double(), eps), P.rms_norm(k, wk.double(), eps)
    qn = torch.cat([P.rope_neox(qn[..., :rot], cos, sin), qn[..., rot:]], -1)
    kn = torch.cat([P.rope_neox(kn[..., :rot], cos, sin), kn[..., rot:]], -1)
    got = x.double().cpu()
    assert torch.allclose(got[:, :H * D].reshape(T, H, D), qn, **tol(dt))
    assert torch.allclose(got[:, H * D:(H + Hkv) * D].reshape(T, Hkv, D), kn, **tol(dt))
    assert torch.equal(got[:, (H + Hkv) * D:], qkv[:, (H + Hkv) * D:].double())      # v and the padding untouched
    c = cache.double().cpu()
    want_c = torch.zeros_like(c)
    for t in range(T):
        s = int(slots[t])
        if s >= 0:
            want_c[s // bs, 0, :, s % bs] = kn[t]
            want_c[s // bs, 1, :, s % bs] = v[t]
    assert torch.allclose(c, want_c, **tol(dt))


def paged_case(rng, reqs, H, Hkv, D, bs, dt, extra_blocks=3, window=None):
    """reqs = [(history, new)].  Returns the kernel's inputs and the plain answer [T, H, D].

    With ``window`` the pages that the window has passed before this step are gone, as the cache manager leaves
    them: a page wholly below ``history - window + 1`` has the table entry -1 and its keys are nowhere; every page
    no request holds (page 0 among them, where a kernel that mistook -1 for a page id might look) is NaN, so a
    kernel that reads a key it must not see shows."""
    g = torch.Generator().manual_seed(rng.randrange(1 << 30))
    total_blocks = sum((h + n + bs - 1) // bs for h, n in reqs) + extra_blocks
    perm = list(range(1 if window else 0, total_blocks))
    rng.shuffle(perm)
    cache = (torch.randn(total_blocks, 2, Hkv, bs, D, generator=g) * 50).to(dt)   # garbage where nothing is stored
    if window:
        cache[:] = float("nan")
    max_blocks = max((h + n + bs - 1) // bs for h, n in reqs) + 1
    table = torch.full((len(reqs), max_blocks), -1, dtype=torch.int32)
    qs, ks, vs, pos, cu = [], [], [], [], [0]
    for b, (hist, new) in enumerate(reqs):
        L = hist + new
        k = torch.randn(L, Hkv, D, generator=g).to(dt)
        v = torch.randn(L, Hkv, D, generator=g).to(dt)
        q = torch.randn(new, H, D, generator=g).to(dt)
        first = max(0, hist - window + 1) // bs if window else 0      # pages before it were given back
        for i in range(first, (L + bs - 1) // bs):
            blk = perm.pop()
            table[b, i] = blk
            n = min(bs, L - i * bs)
            cache[blk] = (torch.randn(2, Hkv, bs, D, generator=g) * 50).to(dt)    # what an earlier holder left
            cache[blk, 0, :, :n] = k[i * bs:i * bs + n].transpose(0, 1)
            cache[blk, 1, :, :n] = v[i * bs:i * bs + n].transpose(0, 1)
        qs.append(q); ks.append(k); vs.append(v)
        pos += list(range(hist, L))
        cu.append(cu[-1] + new)
    return (torch.cat(qs), cache, table, torch.tensor(cu, dtype=torch.int32), torch.tensor(pos, dtype=torch.int32),
            qs, ks, vs)


def plain_paged(reqs, qs, ks, vs, scale, window=None):
    outs = []
    for (hist, new), q, k, v in zip(reqs, qs, ks, vs):
        qfull = torch.cat([torch.zeros(hist, *q.shape[1:], dtype=torch.float64), q.double()])
        outs.append(P.causal_gqa_attention(qfull, k.double(), v.double(), scale, window)[hist:])
    return torch.cat(outs)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H,Hkv,D,bs,window", [(4, 1, 16, 4, None), (6, 2, 32, 16, None), (5, 5, 48, 8, 7),
                                                (8, 2, 128, 16, None), (3, 1, 80, 16, 33), (2, 2, 256, 32, None)])
def test_attention_generic(dt, H, Hkv, D, bs, window):
    from dinfer_b200.kernels import ops
    rng = random.Random(H * 1000 + D)
    reqs = [(40, 5), (70, 1), (0, 33), (130, 64), (0, 1), (7, 1)]        # portions with history beside decodes
    q, cache, table, cu, pos, qs, ks, vs = paged_case(rng, reqs, H, Hkv, D, bs, dt, window=window)
    scale = D ** -0.5
    out = torch.empty(q.shape[0], H * D, dtype=dt, device="cuda")
    ops.attention_generic(dev(q).reshape(-1, H * D), out, dev(cache), dev(table), dev(cu), dev(pos), H, Hkv, D,
                          scale, window or 0)
    want = plain_paged(reqs, qs, ks, vs, scale, window).reshape(-1, H * D)
    assert torch.allclose(out.double().cpu(), want, **tol(dt))


def test_attention_finds_a_far_key():
    """One key among hundreds, on another page, is made to dominate: the output must be its value."""
    from dinfer_b200.kernels import ops
    rng = random.Random(9)
    H, Hkv, D, bs = 4, 2, 64, 16
    reqs = [(600, 1), (300, 2)]
    q, cache, table, cu, pos, qs, ks, vs = paged_case(rng, reqs, H, Hkv, D, bs, torch.float32)
    far = 37                                                  # position of the key that must win, request 0
    q[0] = 0
    q[0, :, 0] = 100.0
    blk = int(table[0, far // bs])
    cache[:, 0, :, :, 0] = 0                                  # no other key has weight along dim 0
    cache[blk, 0, :, far % bs, 0] = 10.0
    out = torch.empty(q.shape[0], H * D, device="cuda")
    ops.attention_generic(dev(q).reshape(-1, H * D), out, dev(cache), dev(table), dev(cu), dev(pos), H, Hkv, D, 1.0, 0)
    got = out[0].reshape(H, D).cpu()
    want = cache[blk, 1, :, far % bs].repeat_interleave(H // Hkv, 0)
    assert torch.allclose(got, want, atol=1e-5)


@pytest.mark.parametrize("V", [517, 4099, 151936])
def test_argmax_and_sampling(V):
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(V)
    R = 6
    logits = torch.randn(R, V, generator=g) * 3
    logits[2, 11] = logits[2, 400] = 50.0                     # a tie: the lower index wins
    d = dev(logits)
    assert S.argmax(d).cpu().tolist() == [int(torch.argmax(logits[i])) if i != 2 else 11 for i in range(R)]
    temps = torch.tensor([0.0, 0.7, 1.0, 1.3, 0.8, 1.0])
    topk = torch.tensor([-1, -1, 5, -1, 40, 3], dtype=torch.int32)
    topp = torch.tensor([1.0, 1.0, 1.0, 0.6, 0.9, 0.5])
    minp = torch.tensor([0.0, 0.0, 0.0, 0.0, 0.02, 0.0])
    agree = total = 0
    for off in range(25):
        seeds = torch.tensor([7, 8, 9, 10, 11, 12], dtype=torch.int64)
        offs = torch.full((R,), off, dtype=torch.int64)
        got = S.sample(d, dev(temps), dev(seeds), dev(offs), top_k=dev(topk), top_p=dev(topp), min_p=dev(minp)).cpu()
        for i in range(R):
            want = P.sample_token(logits[i], float(temps[i]), int(seeds[i]), off, int(topk[i]), float(topp[i]),
                                  float(minp[i]))
            total += 1
            agree += int(got[i]) == want
    # f32 sums against f64: a draw that lands within rounding of a boundary may pick the neighbour
    assert agree >= total - 2, f"{agree}/{total}"


@pytest.mark.parametrize("R,V,ld", [(64, 151936, 151936), (41, 517, 517), (100, 4099, 4104), (40, 1000, 1001)])
def test_argmax_of_many_rows(R, V, ld):
    """From 40 rows on the argmax runs a CTA per row: every row, ties to the lowest index, rows that start on no
    16-byte boundary, a vocabulary that is no multiple of four, columns beyond the vocabulary ignored."""
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(R + V)
    full = torch.randn(R, ld, generator=g) * 3
    full[:, V:] = 1e9                                         # beyond the vocabulary: must not be looked at
    logits = full[:, :V]
    logits[3, 5] = logits[3, V - 1] = 60.0                    # a tie: the lower index wins
    logits[7, V - 1] = 70.0                                   # the last column
    logits[8, 0] = 70.0
    got = S.argmax(dev(full)[:, :V]).cpu().tolist()
    want = [int(torch.argmax(logits[i])) for i in range(R)]
    want[3] = 5
    assert got == want


def test_sampling_distribution_and_batch_independence():
    from dinfer_b200.sampling import sampler as S
    logits = torch.tensor([[2.0, 1.0, 0.5, -1.0, 3.0, 0.0, -30.0]])
    n = 3000
    d = dev(logits.repeat(n, 1))
    temps = dev(torch.full((n,), 0.8))
    seeds = dev(torch.full((n,), 123, dtype=torch.int64))
    offs = dev(torch.arange(n, dtype=torch.int64))
    got = S.sample(d, temps, seeds, offs).cpu()
    freq = torch.bincount(got.long(), minlength=7).double() / n
    want = torch.softmax(logits[0].double() / 0.8, 0)
    assert float((freq - want).abs().max()) < 0.03
    # the same (seed, offset) gives the same token wherever the row stands in the batch
    perm = torch.randperm(n)
    got2 = S.sample(d, temps, seeds, dev(torch.arange(n, dtype=torch.int64)[perm])).cpu()
    assert torch.equal(got2, got[perm])


def test_penalties():
    from dinfer_b200.sampling import sampler as S
    V = 50
    logits = torch.linspace(-2, 2, V).repeat(2, 1)
    ids = torch.tensor([3, 40, 40, 7, 40, 3,   1, 2], dtype=torch.int32)     # row 0: prompt [3, 40], output [40, 7, 40, 3]
    offsets = torch.tensor([0, 6, 8], dtype=torch.int32)
    plen = torch.tensor([2, 2], dtype=torch.int32)
    rep, freq, pres = torch.tensor([1.5, 1.0]), torch.tensor([0.3, 0.0]), torch.tensor([0.2, 0.0])
    d = dev(logits.clone())
    S.apply_penalties(d, dev(ids), dev(offsets), dev(plen), dev(rep), dev(freq), dev(pres))
    want = torch.stack([P.penalties(logits[0], [3, 40], [40, 7, 40, 3], 1.5, 0.3, 0.2),
                        P.penalties(logits[1], [1, 2], [], 1.0, 0.0, 0.0)])
    assert not torch.equal(want[0], logits[0]) and torch.equal(want[1], logits[1])
    assert torch.allclose(d.cpu(), want, atol=1e-6)


@pytest.mark.parametrize("V,ld", [(517, 517), (151936, 151936), (1000, 1024)])
@pytest.mark.parametrize("k", [0, 5, 32])
def test_logprobs_and_logit_bias(V, ld, k):
    """Log-probabilities of the chosen token, its rank and the k most likely tokens against log_softmax / topk;
    ties go to the lower id; additive biases land on the given (row, token) pairs only."""
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(V + k)
    R = 5
    full = (torch.randn(R, ld, generator=g) * 4).cuda()
    logits = full[:, :V]
    logits[1, 7] = logits[1, 3] = float(logits[1].max()) + 1.0          # a tie at the top: id 3 comes first
    logits[2, V - 1] = float("-inf")
    chosen = torch.tensor([0, 7, V - 2, 11, V // 2], dtype=torch.int32, device="cuda")
    ids, lp, rank = S.logprobs(logits, chosen, k)
    want = torch.log_softmax(logits.double(), dim=-1)
    for r in range(R):
        c = int(chosen[r])
        assert int(ids[r, 0]) == c and abs(float(lp[r, 0]) - float(want[r, c])) < 1e-4
        assert int(rank[r]) == int((logits[r] > logits[r, c]).sum())
        if k:
            order = sorted(range(V), key=lambda i: (-float(logits[r, i]), i))[:k]
            assert ids[r, 1:].tolist() == order
            assert torch.allclose(lp[r, 1:].double().cpu(), want[r, order].cpu(), atol=1e-4)
    assert ids[1, 1:3].tolist() == [3, 7][:k] if k else True
    before = logits.clone()
    rows = torch.tensor([0, 0, 3, 4], dtype=torch.int32, device="cuda")
    toks = torch.tensor([1, V - 1, 5, 0], dtype=torch.int32, device="cuda")
    bias = torch.tensor([2.5, -100.0, 100.0, 0.25], device="cuda")
    S.logit_bias(logits, rows, toks, bias)
    want_b = before.clone()
    for r_, t_, b_ in zip(rows.tolist(), toks.tolist(), bias.tolist()):
        want_b[r_, t_] += b_
    assert torch.equal(logits, want_b)
    assert torch.equal(full[:, V:], full[:, V:])                        # the padding of the rows is untouched


def test_top_k_the_short_way_and_its_fallbacks():
    """A small k takes the candidate list, a large one or a crowded bin the radix descent; fewer kept entries than
    k keep them all.  Every way must keep the same set as the plain sampler: same tokens for the same draws."""
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(77)
    V = 20011
    rows = []
    base = torch.randn(V, generator=g) * 3
    rows.append((base.clone(), 512, 1.0, 0.0))                 # the largest k of the short way
    rows.append((base.clone(), 513, 0.9, 0.0))                 # just beyond it: radix
    crowded = base.clone()
    crowded[100:6100] = float(base.max()) + 1.0                # 6000 equal values at the top: the bin overflows
    rows.append((crowded, 10, 1.0, 0.0))                       # (all 6000 ties are kept)
    rows.append((base.clone(), 50, 0.7, 0.3))                  # min_p leaves fewer than k
    tied = base.clone()
    tied[[5, 900, 15000]] = float(base.max()) + 2.0            # ties across the k-th place are all kept
    rows.append((tied, 2, 1.0, 0.0))
    rows.append((base.clone(), 1, 0.5, 0.0))
    logits = torch.stack([r[0] for r in rows])
    R = len(rows)
    d = dev(logits)
    temps = torch.full((R,), 0.9)
    topk = torch.tensor([r[1] for r in rows], dtype=torch.int32)
    topp = torch.tensor([r[2] for r in rows])
    minp = torch.tensor([r[3] for r in rows])
    agree = total = 0
    for off in range(30):
        seeds = torch.arange(R, dtype=torch.int64) + 3
        offs = torch.full((R,), off, dtype=torch.int64)
        got = S.sample(d, dev(temps), dev(seeds), dev(offs), top_k=dev(topk), top_p=dev(topp), min_p=dev(minp)).cpu()
        for i in range(R):
            want = P.sample_token(logits[i], float(temps[i]), int(seeds[i]), off, int(topk[i]), float(topp[i]),
                                  float(minp[i]))
            total += 1
            agree += int(got[i]) == want
    assert agree >= total - 2, f"{agree}/{total}"
    got = S.sample(d, dev(temps), dev(seeds), dev(offs), top_k=dev(topk), top_p=dev(topp), min_p=dev(minp)).cpu()
    assert int(got[5]) == int(torch.argmax(base)) and int(got[4]) in (5, 900, 15000)
    # top-p over thousands of exact ties: the threshold keeps all entries of a value or none (as the reference's
    # kernel does, crates/kernels/cuda/sampling.cu:99-124), where a sort would cut through them
    topp2 = topp.clone()
    topp2[2] = 0.8
    seen = set()
    for off in range(40):
        offs = torch.full((R,), off, dtype=torch.int64)
        seen.add(int(S.sample(d, dev(temps), dev(seeds), dev(offs), top_k=dev(topk), top_p=dev(topp2), min_p=dev(minp)).cpu()[2]))
    assert all(100 <= t < 6100 for t in seen) and max(seen) > 100 + 0.9 * 6000


@pytest.mark.parametrize("V", [7, 40, 8 * 1024 + 3, 151936])
def test_sampling_cuts_and_many_rows(V):
    """Rows whose thresholds lie at the first cuts, in a gap far below the maximum (one certain token), among more entries
    than the short way takes, between masked entries, across ties; one row at a time and 24 at once: the draw falls into the
    token's share of the plain sampler's mass, the same tokens both ways."""
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(V)
    base = torch.randn(V, generator=g) * 2
    sure = base - 80.0
    sure[V // 3] = 60.0                                       # everything else 130 and more below
    spread = torch.linspace(-400.0, 20.0, V)[torch.randperm(V, generator=g)]
    masked = base.clone()
    masked[torch.randperm(V, generator=g)[:V - max(2, V // 50)]] = float("-inf")
    ties = base.round()
    flat = base * 0.01
    rows = [(r, k, p, mp) for r in (base, sure, spread, masked, flat)
            for k, p, mp in ((-1, 0.9, 0.0), (min(20, max(1, V // 2)), 1.0, 0.0), (5, 0.7, 0.0), (-1, 0.999, 1e-4))]
    rows += [(ties, k, 1.0, mp) for k, mp in ((-1, 0.0), (20, 0.0), (5, 0.1), (600, 0.0))]
    logits = torch.stack([r[0] for r in rows])
    R = len(rows)
    assert R >= 19
    temps = torch.full((R,), 0.8)
    topk = torch.tensor([r[1] for r in rows], dtype=torch.int32)
    topp, minp = torch.tensor([r[2] for r in rows]), torch.tensor([r[3] for r in rows])
    seeds = torch.arange(R, dtype=torch.int64) + 11
    d, cols = dev(logits), [dev(t) for t in (temps, seeds, topk, topp, minp)]
    for off in range(6):
        offs = dev(torch.full((R,), off, dtype=torch.int64))
        got = S.sample(d, cols[0], cols[1], offs, top_k=cols[2], top_p=cols[3], min_p=cols[4])
        alone = torch.cat([S.sample(d[i:i + 1], cols[0][i:i + 1], cols[1][i:i + 1], offs[i:i + 1], top_k=cols[2][i:i + 1],
                                    top_p=cols[3][i:i + 1], min_p=cols[4][i:i + 1]) for i in range(R)])
        assert torch.equal(got, alone)
        for i in range(R):
            # the token's share of the cumulative mass holds the draw: a sum over a segment, its warp, the block and the
            # cluster is off by at most (seg + 5 + 32 + 8) 2^-24 of the total, a threshold by an entry at most
            x = P.filter_logits(logits[i].double() / 0.8, int(topk[i]), float(topp[i]), float(minp[i]))
            w = torch.exp(x - x.max())
            t = int(got[i])
            near = float(w.sum()) * 64 * 2.0 ** -24 + 2 * float(w[w > 0].min())
            target, upto = P.philox_uniform(int(seeds[i]), off) * float(w.sum()), float(w[:t + 1].sum())
            assert upto >= target - near and upto - float(w[t]) <= target + near, (i, off)


@pytest.mark.parametrize("V", [3001, 50001, 151936])
def test_sampling_thresholds_far_down_a_row(V):
    """Thresholds below more entries than the short way collects: flat rows (around zero, where floats crowd), rows of few
    distinct values, one value, masked rows with fewer entries than k; nine rows at once and one at a time.  The draw falls
    into the token's share of the plain sampler's mass."""
    from dinfer_b200.sampling import sampler as S
    g = torch.Generator().manual_seed(V + 1)
    base = torch.randn(V, generator=g)
    rounded = (base * 3).bfloat16().float()
    masked = base.clone()
    masked[torch.randperm(V, generator=g)[:V - 1500]] = float("-inf")
    asks = [(-1, 0.5, 0.0), (-1, 0.9, 0.0), (-1, 0.99, 0.0), (-1, 0.999, 1e-3), (1000, 1.0, 0.0), (1000, 0.9, 0.0), (2000, 1.0, 0.0),
            (2000, 0.95, 0.0), (513, 1.0, 0.2)]
    R = len(asks)
    temps, seeds = torch.full((R,), 0.7), torch.arange(R, dtype=torch.int64) + 5
    topk = torch.tensor([a[0] for a in asks], dtype=torch.int32)
    topp, minp = torch.tensor([a[1] for a in asks]), torch.tensor([a[2] for a in asks])
    cols = [dev(t) for t in (temps, seeds, topk, topp, minp)]
    for row in (base, base * 3, rounded, masked, base + 20.0, torch.zeros(V)):
        d = dev(row)[None].expand(R, V).contiguous()
        scaled = row.double() / 0.7
        weights = []
        for a in asks:                                        # (a sort cuts through equal values; the kernel keeps all of them)
            x = P.filter_logits(scaled, *a)
            weights.append(torch.where(scaled >= x[x > float("-inf")].min(), torch.exp(scaled - scaled.max()), torch.zeros(())))
        for off in range(4):
            offs = dev(torch.full((R,), off, dtype=torch.int64))
            got = S.sample(d, cols[0], cols[1], offs, top_k=cols[2], top_p=cols[3], min_p=cols[4])
            alone = torch.cat([S.sample(d[i:i + 1], cols[0][i:i + 1], cols[1][i:i + 1], offs[i:i + 1], top_k=cols[2][i:i + 1],
                                        top_p=cols[3][i:i + 1], min_p=cols[4][i:i + 1]) for i in range(R)])
            assert torch.equal(got, alone)
            for i, w in enumerate(weights):
                # as above: sums off by at most (seg + 5 + 32 + 8) 2^-24 of the total, a threshold by an entry at most
                t = int(got[i])
                near = float(w.sum()) * 64 * 2.0 ** -24 + 2 * float(w[w > 0].min())
                target, upto = P.philox_uniform(int(seeds[i]), off) * float(w.sum()), float(w[:t + 1].sum())
                assert upto >= target - near and upto - float(w[t]) <= target + near, (i, off)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_attention_generic_without_pages(dt):
    """A request whose table holds no page (a dummy row of a captured graph) has no keys: its output is zero and
    nothing outside the cache is read; the request beside it is untouched by it."""
    from dinfer_b200.kernels import ops
    H_, Hkv, D, bs = 4, 2, 24, 4
    g = torch.Generator().manual_seed(5)
    cache = dev(torch.randn(6, 2, Hkv, bs, D, generator=g)).to(dt)
    q = dev(torch.randn(2, H_ * D, generator=g)).to(dt)
    out = torch.full((2, H_ * D), float("nan"), dtype=dt, device="cuda")
    table = dev(torch.tensor([[-1, -1], [3, 1]], dtype=torch.int32))
    cu = dev(torch.tensor([0, 1, 2], dtype=torch.int32))
    pos = dev(torch.tensor([0, 5], dtype=torch.int32))
    ops.attention_generic(q, out, cache, table, cu, pos, H_, Hkv, D, D ** -0.5, 0)
    assert torch.equal(out[0].float(), torch.zeros(H_ * D, device="cuda"))
    alone = torch.empty((1, H_ * D), dtype=dt, device="cuda")
    ops.attention_generic(q[1:], alone, cache, table[1:], dev(torch.tensor([0, 1], dtype=torch.int32)), pos[1:],
                          H_, Hkv, D, D ** -0.5, 0)
    assert torch.equal(out[1], alone[0]) and torch.isfinite(out[1].float()).all()


@pytest.mark.parametrize("e", [-100, -112, -120, -126, -135, -149])
@pytest.mark.parametrize("small", ["a", "w"])
@pytest.mark.parametrize("other", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M, N, K", [(40, 72, 96), (200, 40, 1001)])
def test_gemm_f32_small_elements(e, small, other, M, N, K):
    """Elements far down the range of 32-bit numbers, down to the last ones, against ones that bring the products back up: K
    products summed to 32-bit accuracy are off by at most (K + 1) 2^-24 of the sum of their sizes, wherever the elements lie."""
    from dinfer_b200.kernels import gemm_ops, ops
    g = torch.Generator().manual_seed(M - e)
    tiny = (torch.randn(M if small == "a" else N, K, generator=g, dtype=torch.float64) * 2.0 ** e).float().cuda()
    big = (torch.randn(N if small == "a" else M, K, generator=g, dtype=torch.float64) * 2.0 ** 80).to(other).cuda()
    a, w = (tiny, big) if small == "a" else (big, tiny)
    c = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, c)
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((c.double() - want).abs() <= (K + 1) * 2.0 ** -24 * size).all())
    assert gemm_ops.device_status() == 0


@pytest.mark.parametrize("e, f", [(115, -20), (110, 10), (126, 0)])
def test_gemm_f32_large_elements(e, f):
    """Elements and sums near the top of the range, where the scaled parts are no numbers any more: summed again."""
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(e)
    M, N, K = 50, 40, 96
    a = (torch.rand(M, K, generator=g, dtype=torch.float64) * 2.0 ** e).float().cuda()
    w = (torch.rand(N, K, generator=g, dtype=torch.float64) * 2.0 ** f / K).float().cuda()
    c = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, c)
    want = a.double() @ w.double().T
    assert bool(((c.double() - want).abs() <= (K + 1) * 2.0 ** -24 * want).all())


@pytest.mark.parametrize("M, N, K", [(33, 1, 1), (64, 9, 16), (333, 48, 16), (335, 160, 64), (1000, 48, 33), (2048, 16, 64), (7104, 8, 64), (7105, 8, 64),
                                     (333, 160, 65), (337, 168, 64)])
@pytest.mark.parametrize("a_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
def test_gemm_f32_short_sums(M, N, K, a_dtype, w_dtype):
    """Short sums of more than 32 rows, on either side of the line between a warp a column and tiles; strided rows in and out.  K
    products summed in 32-bit are off by at most (K + 1) 2^-24 of the sum of their sizes."""
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N)
    a, w = torch.randn(M, K + 3, generator=g).to(a_dtype).cuda()[:, 1:K + 1], torch.randn(N, K, generator=g).to(w_dtype).cuda()
    wide = torch.full((M, N + 5), 7.0, device="cuda")
    ops.gemm_f32(a, w, wide[:, 2:N + 2])
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((wide[:, 2:N + 2].double() - want).abs() <= (K + 1) * 2.0 ** -24 * size).all())
    assert bool((wide[:, :2] == 7.0).all()) and bool((wide[:, N + 2:] == 7.0).all())


@pytest.mark.parametrize("M, N", [(33, 1793), (65, 1000), (333, 1024), (2049, 130), (64, 3584)])
@pytest.mark.parametrize("K", [1, 7, 8, 12, 16, 17, 32, 33, 37, 40, 41])
@pytest.mark.parametrize("a_dtype, w_dtype, out", [(torch.float32, torch.float32, torch.float32), (torch.bfloat16, torch.float32, torch.bfloat16),
                                                   (torch.float32, torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("shift", [0, 1])
def test_gemm_f32_short_tiles(M, N, K, a_dtype, w_dtype, out, shift):
    """Short sums of many rows and columns: tiles of multiply-adds up to a line and the tensor cores beyond, edges of a tile, rows
    that take four elements at a time and rows that do not, several problems at once.  K products summed in 32-bit are off by
    at most (K + 1) 2^-24 of the sum of their sizes; a bfloat16 result by 2^-8 of itself more."""
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = (torch.randn(n, (K + 7) // 4 * 4, generator=g).to(t).cuda()[:, shift:K + shift] for n, t in ((M, a_dtype), (N, w_dtype)))
    wide = torch.full((M, (N + 11) // 4 * 4), 7.0, dtype=out, device="cuda")
    ops.gemm_f32(a, w, wide[:, 4:N + 4])
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    bound = (K + 1) * 2.0 ** -24 * size + (2.0 ** -8 * want.abs() if out == torch.bfloat16 else 0)
    assert bool(((wide[:, 4:N + 4].double() - want).abs() <= bound).all())
    assert bool((wide[:, :4] == 7.0).all()) and bool((wide[:, N + 4:] == 7.0).all())


@pytest.mark.parametrize("B, M, N, K", [(3, 70, 200, 16), (5, 33, 8, 24), (2, 300, 130, 40)])
def test_gemm_f32_short_tiles_batched(B, M, N, K):
    from dinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(M, B, K, generator=g).cuda(), torch.randn(B, N, K, generator=g).cuda()
    c = torch.empty(M, B, N, device="cuda")
    ops.gemm_f32_batched(a, w, c)
    want = torch.einsum("mbk,bnk->mbn", a.double(), w.double())
    size = torch.einsum("mbk,bnk->mbn", a.double().abs(), w.double().abs())
    assert bool(((c.double() - want).abs() <= (K + 1) * 2.0 ** -24 * size).all())


def test_gemm_f32_short_sums_that_are_not_finite():
    """Infinities and NaNs reach their own row or column and nothing else."""
    import math
    from dinfer_b200.kernels import ops
    for M, N, K in ((333, 16, 40), (333, 1024, 40), (333, 1024, 200)):
        a, w = torch.ones(M, K, device="cuda"), torch.ones(N, K, device="cuda")
        a[5, 3], w[7, K - 1], a[9, 0] = math.inf, math.nan, -math.inf
        c = torch.empty(M, N, device="cuda")
        ops.gemm_f32(a, w, c)
        assert bool(torch.isnan(c[:, 7]).all())
        c[:, 7] = K
        assert bool((c[5] == torch.where(torch.arange(N, device="cuda") == 7, K, math.inf)).all())
        assert bool((c[9] == torch.where(torch.arange(N, device="cuda") == 7, K, -math.inf)).all())
        c[5], c[9] = K, K
        assert bool((c == K).all())
