"""Portions over expanded latents: the gather, the rotation and the tcgen05 attention alone against plain 64-bit formulas, the
part's two ways against each other, and the expanded way inside captured graphs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def batch(reqs, page, seed):
    """reqs = [(history, new)]: cu, seq, a table of scattered pages and their number."""
    g = torch.Generator().manual_seed(seed)
    per = [(h + n + page - 1) // page for h, n in reqs]
    order = torch.randperm(sum(per) + 3, generator=g).tolist()
    table = torch.full((len(reqs), max(per) + 1), -1, dtype=torch.int32)
    for i, k in enumerate(per):
        table[i, :k] = torch.tensor([order.pop() for _ in range(k)], dtype=torch.int32)
    cu = torch.tensor([0] + [n for _, n in reqs], dtype=torch.int32).cumsum(0).to(torch.int32)
    seq = torch.tensor([h + n for h, n in reqs], dtype=torch.int32)
    return cu, seq, table, sum(per) + 3


CASES = [  # D, P, R, H, page, window, sinks, requests
    (128, 64, 512, 2, 16, 0, False, [(0, 2), (0, 127), (5, 128), (0, 129)]),
    (128, 64, 96, 3, 8, 0, True, [(300, 256), (0, 1), (40, 257), (7, 1)]),
    (128, 32, 64, 1, 64, 100, False, [(0, 300), (1000, 130), (90, 12)]),
    (64, 32, 64, 4, 16, 0, False, [(0, 513), (129, 3)]),
    (64, 0, 40, 2, 4, 37, True, [(200, 140), (10, 30), (64, 64)]),
    (64, 64, 64, 1, 16, 128, False, [(0, 600)] + [(16 * i, 2) for i in range(40)]),
]


@pytest.mark.parametrize("case", CASES)
def test_rows_and_attention_against_plain(case):
    from dinfer_b200.kernels import gemm_ops, latent_ops as L
    D, P, R, H, page, window, with_sinks, reqs = case
    g = torch.Generator().manual_seed(D + P + R)
    cu, seq, table, pages = batch(reqs, page, 1)
    cache = torch.randn(pages, 1, 1, page, R + P, generator=g).to(torch.bfloat16)
    T = int(cu[-1])
    q = torch.randn(T, H * (D + P), generator=g).to(torch.bfloat16)
    w = (torch.randn(H * 2 * D, R, generator=g) * R ** -0.5).to(torch.bfloat16)
    sinks = torch.randn(H, generator=g) if with_sinks else None
    portions = [(n, h + n) for h, n in reqs if n > 1]
    rows = L.expanded_rows(portions, window) + 5
    c = lambda t: None if t is None else t.cuda()
    lat = L.latent_rows(c(cache), c(table), c(cu), c(seq), rows, window)
    kv = lat[:, :R] @ c(w).T
    out = torch.full((T, H, D), float("nan"), dtype=torch.bfloat16, device="cuda")
    scale = (D + P) ** -0.5
    L.attention_latent_umma(c(q), out, lat, kv, c(cu), c(seq), R, P, D, scale, window, sinks=c(sinks),
                            pair_bound=sum((n + 255) // 256 for n, _ in portions) + 2)
    gemm_ops.check_status()
    lat, kv, out = lat.cpu(), kv.cpu().double(), out.cpu()
    at = 0
    for i, (h, n) in enumerate(reqs):
        t0 = int(cu[i])
        if n == 1:
            assert bool(torch.isnan(out[t0].float()).all())    # not this kernel's
            continue
        skip = max(0, h - window + 1) if window else 0
        keys = h + n - skip
        j = torch.arange(skip, h + n)
        want = cache[table[i].long()[j // page], 0, 0, j % page]
        assert torch.equal(lat[at:at + keys], want)
        filled = (keys + 127) // 128 * 128
        assert bool((lat[at + keys:at + filled] == 0).all())
        K = kv[at:at + keys].reshape(keys, H, 2, D)
        for hd in range(H):
            qh = q[t0:t0 + n, hd * (D + P):(hd + 1) * (D + P)].double()
            s = (qh[:, :D] @ K[:, hd, 0].T + qh[:, D:] @ want[:, R:].double().T) * scale
            pos = h + torch.arange(n)[:, None]
            seen = (j[None] <= pos) & ((pos - j[None] < window) if window else True)
            s = s.masked_fill(~seen, float("-inf"))
            top = s.max(1, keepdim=True).values
            e = torch.exp(s - top)
            den = e.sum(1, keepdim=True) + (torch.exp(sinks[hd].double() - top) if with_sinks else 0.0)
            p = e / den
            o = p @ K[:, hd, 1]
            # weights rounded to bfloat16 (2^-9 each, against sums that are not), the result (2^-9), scores in 32-bit (an
            # exponential's relative error: a few 1e-6 here)
            bound = (2.0 ** -8) * (p @ K[:, hd, 1].abs()) + 2.0 ** -8 * o.abs() + 1e-5
            assert bool(((out[t0:t0 + n, hd].double() - o).abs() <= bound).all())
        at += filled
    assert bool((lat[at:] == 0).all())


@pytest.mark.parametrize("D,P,H,window,with_sinks,reqs,shared", [
    (128, 64, 3, 0, True, [(0, 640)], False), (128, 64, 2, 0, False, [(0, 641), (0, 1), (500, 129), (0, 30)], True),
    (64, 32, 4, 0, True, [(5000, 257)], True), (128, 64, 1, 900, False, [(2000, 300), (10, 700)], True),
    (128, 16, 16, 0, False, [(0, 1100)], False), (64, 64, 1, 0, False, [(639, 2), (640, 128), (767, 2)], True),
    (128, 64, 3, 0, True, [(0, 700)], True), (128, 16, 8, 0, False, [(0, 1100)], True),
    (128, 64, 16, 0, False, [(0, 2048)], True), (128, 32, 12, 0, True, [(1500, 2100), (0, 3)], True)])
def test_two_ctas_to_a_pair(D, P, H, window, with_sinks, reqs, shared):
    """Row-tile pairs whose keys two CTAs share, beside pairs too short for it, pairs with one row tile, one row of one, an odd number of
    key tiles, histories and windows, launches whose CTAs all run at once and launches of more (and two batches whose keys are
    not shared): the same as without (which the test above holds to the formula), up to the other order of sums and the other
    maximum that weights are rounded against."""
    from dinfer_b200.kernels import gemm_ops, latent_ops as L
    g = torch.Generator().manual_seed(D + H)
    cu, seq, table, pages = batch(reqs, 16, 1)
    R, T = 64, int(cu[-1])
    c = lambda t: None if t is None else t.cuda()
    cache = torch.randn(pages, 1, 1, 16, R + P, generator=g).to(torch.bfloat16).cuda()
    q = (torch.randn(T, H * (D + P), generator=g) * 1.5).to(torch.bfloat16).cuda()
    w = (torch.randn(H * 2 * D, R, generator=g) * R ** -0.5).to(torch.bfloat16).cuda()
    sinks = c(torch.randn(H, generator=g)) if with_sinks else None
    portions = [(n, h + n) for h, n in reqs if n > 1]
    lat = L.latent_rows(cache, c(table), c(cu), c(seq), L.expanded_rows(portions, window), window)
    kv = lat[:, :R] @ w.T
    pairs = sum((n + 255) // 256 for n, _ in portions)
    assert not L.shares_keys(H, pairs, window, 0) and L.shares_keys(H, pairs, window, int(seq.max())) is shared
    got = []
    for longest in (0, int(seq.max())):
        out = torch.full((T, H, D), float("nan"), dtype=torch.bfloat16, device="cuda")
        L.attention_latent_umma(q, out, lat, kv, c(cu), c(seq), R, P, D, (D + P) ** -0.5, window, sinks=sinks, pair_bound=pairs, max_keys=longest)
        gemm_ops.check_status()
        got.append(out.float())
    for i, (h, n) in enumerate(reqs):
        a, b = (o[int(cu[i]):int(cu[i]) + n] for o in got)
        if n == 1:
            assert bool(torch.isnan(b).all())
            continue
        # every weight and every result rounded to bfloat16 once more on either side: 2^-8 of the values' sizes
        assert bool(((a - b).abs() <= 2.0 ** -7 * (a.abs() + kv.float().abs().max() * 0.25)).all())
        assert float((a - b).norm() / a.norm()) < 4e-3


@pytest.mark.parametrize("rows,pairs,bad", [(512, 3, False), (511, 3, True), (256, 3, True), (512, 2, True), (600, 7, False)])
def test_portions_beyond_the_launch_leave_a_status(rows, pairs, bad):
    """Portions that need 512 gathered rows and three row-tile pairs: a launch made for fewer says so."""
    from dinfer_b200.kernels import gemm_ops, latent_ops as L
    from dinfer_b200.kernels.lib import KernelError
    D, P, R, H = 64, 32, 64, 2
    # 256, 128 and 128 gathered rows, a pair each; behind 40 single tokens the scan takes a second turn
    reqs = [(100, 150)] + [(5, 1)] * 40 + [(0, 120), (0, 9)]
    cu, seq, table, pages = batch(reqs, 16, 2)
    c = lambda t: t.cuda()
    cache = torch.randn(pages, 1, 1, 16, R + P).to(torch.bfloat16).cuda()
    q = torch.randn(int(cu[-1]), H * (D + P)).to(torch.bfloat16).cuda()
    w = torch.randn(H * 2 * D, R).to(torch.bfloat16).cuda()
    out = torch.zeros(int(cu[-1]), H, D, dtype=torch.bfloat16, device="cuda")
    lat = L.latent_rows(cache, c(table), c(cu), c(seq), rows, 0)
    L.attention_latent_umma(q, out, lat, lat[:, :R] @ w.T, c(cu), c(seq), R, P, D, 0.1, 0, pair_bound=pairs)
    if bad:
        with pytest.raises(KernelError, match="status 37"):
            gemm_ops.check_status()
        assert gemm_ops.reset_status() == 37
    gemm_ops.check_status()


@pytest.mark.parametrize("P,rot,halves", [(64, 64, False), (32, 20, False), (64, 64, True), (16, 8, True)])
def test_rotation_in_place(P, rot, halves):
    from dinfer_b200.kernels import latent_ops as L
    T, H, D, R = 7, 3, 64, 16
    g = torch.Generator().manual_seed(P + rot)
    q = torch.randn(T, H * (D + P), generator=g).to(torch.bfloat16).cuda()
    pos = torch.randint(0, 50, (T,), generator=g).to(torch.int32).cuda()
    a = torch.rand(50, rot // 2, generator=g) * 6.3
    table = torch.cat([a.cos(), a.sin()], 1).cuda()
    want = torch.zeros(T, H, R + P, dtype=torch.bfloat16, device="cuda")
    L.latent_q_rope(q, pos, table, want, H, D, P, R, halves=halves)
    got = q.clone()
    L.latent_q_turn(got, pos, table, H, D, P, halves=halves)
    assert torch.equal(got.view(T, H, D + P)[:, :, D:], want[:, :, R:])
    assert torch.equal(got.view(T, H, D + P)[:, :, :D], q.view(T, H, D + P)[:, :, :D])


def part_and_context(reqs, window=None, gate=False, sink=False, D=128, P=64, seed=3):
    import dinfer_b200.models.decoder  # noqa: F401
    from dinfer_b200.cache.manager import CacheManager, GroupSpec
    from dinfer_b200.engine.batch import PlanBuilder, StepEntry
    from dinfer_b200.parts.base import MIXERS, BuildEnv, CacheBinding
    from dinfer_b200.parts.spec import PartSpec
    g = torch.Generator().manual_seed(seed)
    h = 256
    params = {"num_heads": 2, "nope_dim": D, "rope_dim": P, "v_dim": D, "kv_rank": 96, "q_rank": 64, "eps": 1e-6, "window": window,
              "position": PartSpec("rope", {"head_dim": P, "rotary_dim": P, "theta": 500.0, "max_positions": 2048,
                                            "style": "interleaved"})}
    if gate:
        params["gate_proj"] = "gate"
    if sink:
        params["sink"] = "sink"
    part = MIXERS.get("latent_attention")(params, BuildEnv(torch.device("cuda"), torch.bfloat16, h, 2048), "")
    part.bind({d.name: ((1 + 0.1 * torch.randn(d.shape, generator=g)) if d.init == "ones"
                        else torch.randn(d.shape, generator=g) * d.shape[-1] ** -0.5).to(torch.bfloat16).cuda() for d in part.declare()})
    pages = sum((a + n + 15) // 16 for a, n in reqs) + 2
    m = CacheManager([GroupSpec(window)], 16, pages, len(reqs) + 1)
    entries = []
    for i, (a, n) in enumerate(reqs):
        assert m.allocate(i, a + n)
        m.advance(i, a)
        entries.append(StepEntry(i, [0] * n, []))
    _, _, ctx = PlanBuilder(m, "cuda", 4096, len(reqs) + 1, 256).build(entries, [a for a, _ in reqs])
    kv = torch.randn(pages, 1, 1, 16, 96 + P, generator=g).to(torch.bfloat16).cuda()
    x = torch.randn(sum(n for _, n in reqs), h, generator=g).to(torch.bfloat16).cuda()
    return part, ctx, CacheBinding(kv=kv, group=0, write=True), x


ABSORBED, EXPANDED = (1e30, 1e30, 0.0, 1.0, 1.0, 1.0, 1.0), (1.0, 1.0, 1.0, 1e30, 1e30, 0.0, 0.0)


@pytest.mark.parametrize("reqs,window,gate,sink", [([(0, 300)], None, False, False), ([(40, 1), (0, 129), (500, 1), (300, 64)], None, True, True),
                                                   ([(700, 150), (3, 1), (0, 2)], 128, False, True)])
def test_both_ways_of_the_part_agree(reqs, window, gate, sink, monkeypatch):
    """The rule's two answers on the same step, single tokens beside portions: two roundings of bfloat16 apart, the same cache."""
    import dataclasses
    from dinfer_b200.parts.latent_attention import LatentAttention
    outs, caches = [], []
    for rates in (ABSORBED, EXPANDED):                                        # one way is free, then the other
        part, ctx, cache, x = part_and_context(reqs, window, gate, sink)
        monkeypatch.setattr(LatentAttention, "RATES", rates)
        shape = part._expanded(ctx, torch.bfloat16)
        assert (shape is None) == (rates is ABSORBED)
        outs.append(part.forward(x, dataclasses.replace(ctx, derived={}), cache).float())
        caches.append(cache.kv.clone())
    assert torch.equal(caches[0], caches[1]) and bool(torch.isfinite(outs[1]).all())
    assert float((outs[0] - outs[1]).norm() / outs[0].norm()) < 1e-2
    # what a request's rows hold does not depend on what lies in another request's pages
    if len(reqs) > 1:
        part, ctx, cache, x = part_and_context(reqs, window, gate, sink)
        table = ctx.groups[0].block_table
        own = set(table[1].tolist())
        for b in table[0].tolist():
            if b >= 0 and b not in own:
                cache.kv[b] = float("inf")
        got = part.forward(x, dataclasses.replace(ctx, derived={}), cache).float()
        a, z = reqs[0][1], reqs[0][1] + reqs[1][1]
        assert torch.equal(got[a:z], outs[1][a:z])


@pytest.mark.parametrize("reqs,rows", [([(0, 129), (500, 1), (40, 1)], 2), ([(500, 1), (0, 129), (0, 2), (40, 1), (3, 7)], 133), ([(9, 1), (0, 300)], 1)])
def test_the_absorbing_products_see_the_single_tokens_only(reqs, rows, monkeypatch):
    """Beside portions over expanded latents: the rows from the first single token to the last."""
    from dinfer_b200.parts.latent_attention import LatentAttention
    monkeypatch.setattr(LatentAttention, "RATES", EXPANDED)
    monkeypatch.setattr(LatentAttention, "MIXED_HOST", 0.0, raising=False)
    seen, absorb = [], LatentAttention.absorb
    monkeypatch.setattr(LatentAttention, "absorb", lambda self, a, w, out: (seen.append((a.shape[0], out.shape[0])), absorb(self, a, w, out))[1])
    part, ctx, cache, x = part_and_context(reqs)
    y = part.forward(x, ctx, cache)
    assert seen == [(rows, rows)] * 2 and bool(torch.isfinite(y.float()).all())


@pytest.mark.parametrize("order", [(0, 1, 2), (1, 0, 2), (1, 2, 0)])
def test_few_single_tokens_beside_a_long_portion(order):
    """Decoded tokens beside a portion share their keys many ways: the workspace follows their number, not the portion's, and
    the portion's rows stay as they are.  Against plain 64-bit formulas."""
    from dinfer_b200.kernels import latent_ops as L
    R, P, H, page, scale = 128, 32, 4, 16, 0.1
    reqs = [[(0, 3000), (3999, 1), (130, 1)][i] for i in order]
    cu, seq, table, pages = batch(reqs, page, 5)
    T = int(cu[-1])
    g = torch.Generator().manual_seed(9)
    cache = torch.randn(pages, 1, 1, page, R + P, generator=g).to(torch.bfloat16)
    q = torch.randn(T, H, R + P, generator=g).to(torch.bfloat16)
    out = torch.full((T, H, R), 7.0, dtype=torch.bfloat16, device="cuda")
    args = (q.cuda(), out, cache.cuda(), table.cuda(), cu.cuda(), seq.cuda())
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    L.attention_latent_tc(*args, R, P, scale, max_q_len=3000, max_seq_len=4000, singles=True)
    # at most 64 ways: sums of R and two numbers for each of 3 requests' heads
    assert torch.cuda.max_memory_allocated() - held <= 2 * 3 * H * 64 * (R + 2) * 4 + 4096
    out = out.cpu()
    for i, (h, n) in enumerate(reqs):
        t0 = int(cu[i])
        if n > 1:
            assert bool((out[t0:t0 + n] == 7.0).all())
            continue
        j = torch.arange(h + 1)
        rows = cache[table[i].long()[j // page], 0, 0, j % page].double()
        p = torch.softmax(q[t0].double() @ rows.T * scale, dim=1)
        o = p @ rows[:, :R]
        # weights rounded to bfloat16 (2^-9 each, against sums that are not), the result (2^-9), scores in 32-bit
        assert bool(((out[t0].double() - o).abs() <= 2.0 ** -8 * (p @ rows[:, :R].abs()) + 2.0 ** -8 * o.abs() + 1e-5).all())


def test_captured_steps_run_over_expanded_latents_too(monkeypatch):
    """Prompts taken in portions of the whole budget beside decoded tokens, kernel by kernel and as graphs: the same logits
    up to rounding, and the graph's bounds hold prompts of other lengths than it was captured on."""
    from dinfer_b200.config.engine_config import EngineConfig
    from dinfer_b200.engine.batch import StepEntry
    from dinfer_b200.engine.runner import ModelRunner
    from dinfer_b200.parts.latent_attention import LatentAttention
    from dinfer_b200.weights.random_init import RandomSource
    mixer = {"heads": 2, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 64, "q_rank": 64, "scale": 96 ** -0.5,
             "rot": {"base": 10000.0, "dims": 32}}
    cfg = {"architecture": "Dobedra", "vocab": 256, "width": 128, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
           "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": 128}}] * 2}
    monkeypatch.setattr(LatentAttention, "RATES", EXPANDED)
    calls = []
    whole = LatentAttention.attend_expanded
    monkeypatch.setattr(LatentAttention, "attend_expanded", lambda self, *a: (calls.append(torch.cuda.is_current_stream_capturing()), whole(self, *a))[1])
    got = []
    for graphs in (False, True):
        runner = ModelRunner(cfg, RandomSource(cfg, 5, std=0.1), EngineConfig(
            max_model_len=512, max_num_seqs=4, max_num_batched_tokens=128, num_blocks=160, block_size=16, dtype="bfloat16",
            enable_cuda_graph=graphs))
        runner.step([StepEntry("d", list(range(40)), [])])
        out = []
        for rnd in range(4):
            for start, n in ((0, 128), (128, 128), (256, 100), (356, 50)):
                logits = runner.step([StepEntry(("p", rnd), [(3 * i + start + rnd) % 256 for i in range(n)], [n - 1]),
                                      StepEntry("d", [rnd + 7], [0])])
                out.append(logits.clone())
            runner.finish(("p", rnd))
        runner.check_device_status()
        got.append(torch.stack(out).float())
    assert any(calls) and not all(calls)
    assert bool(torch.isfinite(got[1]).all())
    assert float((got[0] - got[1]).norm() / got[0].norm()) < 2e-2
