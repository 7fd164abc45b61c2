"""The delta rule in chunks of 32 tokens against the recurrence in 64-bit, no further off than the token loop."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def plain(q, k, v, beta, g, S):
    """One request: q, k [n, H, dk], v [n, H, dv], beta, g [n, H], S [H, dk, dv], 64-bit."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = g[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out, S


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


CASES = [  # H, G, dk, dv, tokens of the requests, fresh, decays, keys
    (2, 1, 128, 128, [200], [1], "mixed", "random"),
    (4, 2, 64, 64, [1, 31, 32, 33, 64, 7], [1, 0, 1, 0, 0, 1], "mixed", "random"),
    (3, 3, 128, 16, [65, 2, 97], [0, 1, 0], "slow", "random"),
    (2, 2, 64, 48, [130], [0], "fast", "random"),
    (2, 1, 128, 32, [96, 50], [1, 0], "zero", "random"),
    (2, 1, 64, 32, [150], [0], "slow", "alike"),
    (2, 2, 128, 256, [40] * 13, [1, 0] * 6 + [1], "mixed", "random"),
]


@pytest.mark.parametrize("case", CASES)
def test_chunks_against_plain(case):
    from dinfer_b200.kernels import delta_ops
    H, G, dk, dv, tokens, fresh, decays, keys = case
    g_ = torch.Generator().manual_seed(dk + dv + len(tokens))
    T, B = sum(tokens), len(tokens)
    rand = lambda *s: torch.randn(*s, generator=g_)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)
    q = unit(rand(T, G, dk)) * dk ** -0.5
    k = unit(rand(T, G, dk) * (0.02 if keys == "alike" else 1.0) + (1.0 if keys == "alike" else 0.0))
    v, beta = rand(T, H, dv), torch.sigmoid(rand(T, H) + (3.0 if keys == "alike" else 0.0))
    x = {"slow": 1e-6 * torch.rand(T, H, generator=g_), "fast": 30 * torch.rand(T, H, generator=g_),
         "mixed": torch.exp(8 * torch.rand(T, H, generator=g_) - 7), "zero": torch.exp(8 * torch.rand(T, H, generator=g_) - 7)}[decays]
    decay = torch.expm1(-x.double()).float()
    if decays == "zero":
        decay[::5] = -1.0                                    # a decay of 0 forgets everything
    state = rand(B + 2, H * dk * dv + 5)
    order = torch.randperm(B + 2, generator=g_)[:B].to(torch.int32)
    cu = torch.tensor([0] + tokens, dtype=torch.int32).cumsum(0).to(torch.int32)
    fr = torch.tensor(fresh, dtype=torch.int32)
    c = lambda t: t.cuda()
    got, states = [], []
    for longest in (0, 1000):
        st = c(state).clone()
        o = delta_ops.recurrence(c(q), c(k), c(v), c(beta), c(decay), st, c(cu), c(order), c(fr), False, longest=longest)
        got.append(o.cpu())
        states.append(st.cpu())
    assert not torch.equal(got[0], got[1])                   # two ways indeed
    rep = H // G
    for i in range(B):
        a, z, slot = int(cu[i]), int(cu[i + 1]), int(order[i])
        S0 = state[slot, :H * dk * dv].double().reshape(H, dk, dv) * (0.0 if fresh[i] else 1.0)
        d = lambda t: t[a:z].double()
        want, S = plain(d(q).repeat_interleave(rep, 1), d(k).repeat_interleave(rep, 1), d(v), d(beta), d(decay) + 1.0, S0)
        for w, loop, chunks in ((want, got[0][a:z], got[1][a:z]),
                                (S, states[0][slot, :H * dk * dv].reshape(H, dk, dv), states[1][slot, :H * dk * dv].reshape(H, dk, dv))):
            # sums of some 200 products in 32-bit: a few 1e-7; the token loop's own error where that is larger
            assert rel(chunks, w) <= 1.5 * rel(loop, w) + 1e-6, (i, rel(chunks, w), rel(loop, w))
    used = set(order.tolist())
    for s in range(B + 2):                                   # other slots and what lies behind S are untouched
        keep = slice(H * dk * dv, None) if s in used else slice(None)
        assert torch.equal(states[1][s, keep], state[s, keep])


def loop_and_chunks(where, value, at):
    """Outputs and states of both ways, one request behind another, with ``value`` in one element of one input at token
    ``at`` of the first request."""
    from dinfer_b200.kernels import delta_ops
    H, G, dk, dv, tokens = 4, 2, 64, 32, [150, 40]
    g = torch.Generator().manual_seed(at + dk)
    T = sum(tokens)
    rand = lambda *s: torch.randn(*s, generator=g)
    x = {"q": rand(T, G, dk) / dk, "k": rand(T, G, dk) * dk ** -0.5, "v": rand(T, H, dv), "beta": torch.sigmoid(rand(T, H)),
         "decay": torch.expm1(-0.1 * torch.rand(T, H, generator=g))}
    x[where].view(T, -1)[at, 1] = value
    state, cu = rand(2, H * dk * dv), torch.tensor([0] + tokens, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32).cuda()
    out = []
    for longest in (0, 1000):
        st = state.clone().cuda()
        o = delta_ops.recurrence(*[x[n].cuda() for n in ("q", "k", "v", "beta", "decay")], st, cu, i32(0, 1), i32(0, 0), False,
                                 longest=longest)
        out.append((o.cpu(), st.cpu().view(2, H, dk, dv)))
    return out


@pytest.mark.parametrize("at", [0, 21, 95, 149])
def test_a_decay_that_is_not_a_number_stays_one(at):
    (loop, loop_state), (chunks, state) = loop_and_chunks("decay", float("nan"), at)
    assert not bool(torch.isfinite(loop[at:150, 1]).any()) and not bool(torch.isfinite(loop_state[0, 1]).any())
    assert not bool(torch.isfinite(chunks[at:150, 1]).any()) and not bool(torch.isfinite(state[0, 1]).any())


@pytest.mark.parametrize("where,value", [(n, x) for n in ("q", "k", "v", "beta", "decay") for x in (float("nan"), float("inf"))][:-1])
@pytest.mark.parametrize("at", [0, 5, 31, 70, 127, 149])
def test_what_is_not_finite_reaches_no_earlier_token(where, value, at):
    """Outputs and states are finite in the same places both ways, and there no further apart than two orders of the sums."""
    for a, b in zip(*loop_and_chunks(where, value, at)):
        fa, fb = torch.isfinite(a), torch.isfinite(b)
        assert torch.equal(fa, fb)
        # sums of some 200 products of a few units in 32-bit
        assert float((a[fa] - b[fa]).abs().max()) < 2e-5 * float(a[fa].abs().max())


def test_sizes_the_chunks_do_not_take_stay_with_the_token_loop():
    from dinfer_b200.kernels import delta_ops
    g = torch.Generator().manual_seed(3)
    for dk, dv in ((32, 32), (64, 24), (128, 40)):
        q, k, v = (torch.randn(60, 1, n, generator=g).cuda() for n in (dk, dk, dv))
        beta, decay = torch.rand(60, 1, generator=g).cuda(), -torch.rand(60, 1, generator=g).cuda()
        outs = []
        for longest in (0, 1000):
            st = torch.zeros(1, dk * dv).cuda()
            i32 = lambda *x: torch.tensor(x, dtype=torch.int32).cuda()
            outs.append(delta_ops.recurrence(q, k, v, beta, decay, st, i32(0, 60), i32(0), i32(1), False, longest=longest))
        assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("lens,runs", [([1] * 64, False), ([1] * 512, False), ([64], False), ([255], False), ([256], True), ([8] * 64, False),
                                       ([16] * 32, True), ([1] * 16 + [240], False), ([1] * 31 + [481], True), ([100, 411], False),
                                       ([1, 2, 470, 64, 9, 3], True)])
def test_which_steps_are_prepared_in_runs(lens, runs):
    """Portions of many tokens; decoded tokens and short portions keep a block per (token, head)."""
    from dinfer_b200.kernels.lib import library
    takes = library("delta_rule").dinfer_delta_prep_runs
    assert bool(takes(sum(lens), len(lens), 8, 128, 4)) is runs
    assert not takes(sum(lens), len(lens), 8, 128, 3) and not takes(sum(lens), len(lens), 8, 32, 4) and not takes(sum(lens), len(lens), 3, 96, 4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,per_channel", [(3, 1, 64, 40, False), (3, 3, 64, 16, True), (2, 1, 128, 72, False)])
def test_preparation_in_runs(dtype, H, G, dk, dv, per_channel):
    """Steps of many tokens (a thread walks eight tokens of a channel) against plain formulas and, beside the short
    steps' kernel, request by request: requests that begin and end anywhere in a run, fresh and carried histories."""
    from dinfer_b200.kernels import delta_ops
    F64 = torch.float64
    g = torch.Generator().manual_seed(dk + dv + H)
    lens, fresh, taps = [1, 2, 470, 64, 9, 3], [1, 0, 1, 0, 0, 1], 4
    T, B, nq, nv = sum(lens), len(lens), G * dk, H * dv
    C, nd = 2 * nq + nv, H * dk if per_channel else H
    Pm = torch.randn(T, C + H + 5, generator=g).to(dtype)
    Am = torch.randn(T, nd, generator=g).to(dtype)
    conv_w, A_log, dt_bias = torch.randn(C, taps, generator=g), torch.randn(H, generator=g), torch.randn(nd, generator=g) - 1.0
    S0 = H * dk * dv
    state = torch.randn(B, S0 + (taps - 1) * C, generator=g)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()
    call = lambda rows, st, cu_, slots, fr: [o.cpu() for o in delta_ops.prep(
        Pm[rows].cuda(), (0, nq, 2 * nq, C + 5), Am[rows].cuda(), conv_w.cuda(), A_log.cuda(), dt_bias.cuda(), st, S0, ints(cu_),
        ints(slots), ints(fr), H, G, dk, dv, taps, per_channel)]
    st = state.clone().cuda()
    got = call(slice(0, T), st, cu, list(range(B)), fresh)
    softplus = lambda z: torch.clamp(z, min=0) + torch.log1p(torch.exp(-z.abs()))
    for i in range(B):
        a, z = int(cu[i]), int(cu[i + 1])
        x = Pm[a:z].to(F64)
        hist = torch.zeros(taps - 1, C, dtype=F64) if fresh[i] else state[i, S0:].to(F64).view(taps - 1, C)
        full = torch.cat([hist, x[:, :C]])
        y = sum(full[d:d + z - a] * conv_w[:, d].to(F64) for d in range(taps))
        y = y * torch.sigmoid(y)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        decay = torch.expm1(-torch.exp(A_log.to(F64)).repeat_interleave(dk if per_channel else 1) * softplus(Am[a:z].to(F64) + dt_bias.to(F64)))
        want = [unit(y[:, :nq].view(-1, G, dk)) * dk ** -0.5, unit(y[:, nq:2 * nq].view(-1, G, dk)), y[:, 2 * nq:].view(-1, H, dv),
                torch.sigmoid(x[:, C + 5:]), decay]
        for o, w in zip(got, want):
            assert torch.allclose(o[a:z].to(F64), w, rtol=2e-5, atol=2e-5)
        assert torch.allclose(st[i, S0:].cpu().to(F64).view(taps - 1, C), full[z - a:], rtol=0, atol=0)
        if z - a < 64:
            alone = call(slice(a, z), state.clone().cuda()[i:i + 1], [0, z - a], [0], [fresh[i]])
            for o, w in zip(got, alone):
                assert torch.allclose(o[a:z], w, rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("B,H,longest,chunks", [(1, 16, 127, False), (1, 16, 128, True), (2, 16, 255, False), (2, 16, 256, True), (3, 16, 511, False),
                                                (3, 16, 512, True), (4, 16, 4000, False)])
def test_which_portions_run_in_chunks(B, H, longest, chunks, monkeypatch):
    from dinfer_b200.kernels import delta_ops
    monkeypatch.setattr(delta_ops, "num_sms", lambda: 148)
    z = lambda *s: torch.zeros(*s, device="cuda")
    i = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    q, v, beta = z(2 * B, 8, 128), z(2 * B, H, 128), z(2 * B, H)
    took = delta_ops._chunks(q, q, v, beta, beta, z(B, H * 128 * 128), i(*range(0, 2 * B + 1, 2)), i(*range(B)), i(*[1] * B),
                             torch.empty_like(v), longest)
    torch.cuda.synchronize()
    assert took is chunks


@pytest.mark.parametrize("dv,H,T", [(16, 3, 11), (32, 5, 7), (64, 1, 1), (64, 3, 43), (128, 16, 9), (128, 1, 5)])
@pytest.mark.parametrize("gate", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_output_norm_of_whole_heads(dv, H, T, gate, out):
    """Four values a lane (a warp's last heads may be past the end), and the same from rows off their alignment."""
    from dinfer_b200.kernels import delta_ops
    g = torch.Generator().manual_seed(dv + T)
    o = torch.randn(T, H, dv, generator=g).cuda()
    heads = H > 1
    w = (1 + 0.2 * torch.randn(H * dv if heads else dv, generator=g)).cuda()
    for sigmoid in (False, True):
        got = []
        for shift in (0, 1):                                 # a row that starts one element in: the other kernel
            z = None if gate is None else torch.randn(T, H * dv + 4, generator=torch.Generator().manual_seed(1)).to(gate)
            if z is not None:
                z = torch.cat([torch.zeros(T, 4 + shift, dtype=gate), z[:, :H * dv], torch.zeros(T, 4 - shift, dtype=gate)], 1).cuda()[:, 4 + shift:4 + shift + H * dv]
            y = torch.empty(T, H * dv + 4, dtype=out, device="cuda")[:, shift:shift + H * dv]
            delta_ops.post(o, w, z, 1e-5, sigmoid, y)
            got.append(y.double().reshape(T, H, dv))
        want = o.double() / torch.sqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5) * w.double().reshape(H if heads else 1, dv)
        if z is not None:
            zz = z.double().reshape(T, H, dv)
            want = want * (torch.sigmoid(zz) if sigmoid else zz * torch.sigmoid(zz))
        # a dozen 32-bit roundings, then one to the output's type
        tol = 12 * 2 ** -23 + (2 ** -8 if out == torch.bfloat16 else 0)
        for y in got:
            assert bool(((y - want).abs() <= tol * want.abs() + 1e-6).all())
