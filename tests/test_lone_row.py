"""A lone token's norm on its way to the product that makes it: what is handed on, and what goes through the norm's own
kernel because the product could not read it as it lies."""
import pytest
import torch

from dinfer_b200.parts.base import BuildEnv, ResidualStream, Unnormed
from dinfer_b200.parts.block import normed
from dinfer_b200.parts.norm import RMSNorm

K = 64


def off(n, dtype, device="cpu", at=1):
    """A contiguous row that starts ``at`` elements behind a 16-byte boundary (0: on it)."""
    return torch.ones(1, n + 8, dtype=dtype, device=device)[:, at:at + n]


class Taker:
    def makes_norm(self, rows):
        return rows == 1


def norm_of(weight, device="cpu"):
    norm = RMSNorm({"size": weight.numel(), "eps": 1e-6}, BuildEnv(torch.device(device), torch.bfloat16, weight.numel(), 16))
    norm.bind({"weight": weight})
    return norm


@pytest.mark.parametrize("at", [0, 1, 4])
@pytest.mark.parametrize("which", ["delta", "weight", "residual"])
def test_rows_off_their_alignment_keep_the_norm_kernel(which, at):
    f32, bf16 = torch.float32, torch.bfloat16
    x, delta, w = off(K, f32, at=0), off(K, bf16, at=0), off(K, bf16, at=0)[0]
    if which == "delta":
        delta = off(K, bf16, at=at)
    elif which == "weight":
        w = off(K, bf16, at=at)[0]
    else:
        x = off(K, f32, at=(at + 1) // 2)
    norm = norm_of(w)
    norm.forward = lambda residual, delta=None, rows=None: "normed"
    got = normed(ResidualStream(x), norm, delta, Taker())
    assert isinstance(got, Unnormed) if at == 0 else got == "normed"


def test_other_types_and_rows_keep_the_norm_kernel():
    norm = norm_of(torch.ones(K, dtype=torch.bfloat16))
    norm.forward = lambda residual, delta=None, rows=None: "normed"
    x = torch.ones(1, K)
    assert isinstance(normed(ResidualStream(x), norm, None, Taker()), Unnormed)
    for stream, delta, taker in ((ResidualStream(x), torch.ones(1, K), Taker()), (ResidualStream(torch.ones(2, K)), None, Taker()),
                                 (ResidualStream(x.bfloat16()), None, Taker()), (ResidualStream(x, results=x), None, Taker()),
                                 (ResidualStream(x), None, None), (ResidualStream(x), None, object())):
        assert normed(stream, norm, delta, taker) == "normed"


@pytest.mark.gpu
@pytest.mark.parametrize("at", [1, 2, 4])
@pytest.mark.parametrize("which", ["delta", "weight"])
def test_a_slice_as_delta_or_weight(which, at):
    """The same block of a feed-forward with a delta or a norm weight that lies off 16 bytes; the way around the norm's kernel may
    round an input of a thousand the other way (2^-8 of it), the product sums 64 of them."""
    from dinfer_b200.parts.mlp import SwiGLU
    env = BuildEnv(torch.device("cuda"), torch.bfloat16, K, 16)
    g = torch.Generator().manual_seed(at)
    ffn = SwiGLU({"intermediate_size": 96}, env, "")
    ffn.bind({d.name: (torch.randn(d.shape, generator=g) * d.shape[-1] ** -0.5).bfloat16().cuda() for d in ffn.declare()})
    delta0, w0, x0 = torch.randn(1, K, generator=g).bfloat16().cuda(), (1 + 0.1 * torch.randn(K, generator=g)).bfloat16().cuda(), torch.randn(1, K, generator=g).cuda()
    results = []
    for shift in (0, at):
        delta, w = off(K, torch.bfloat16, "cuda", shift if which == "delta" else 0), off(K, torch.bfloat16, "cuda", shift if which == "weight" else 0)
        delta.copy_(delta0)
        w.copy_(w0)
        stream = ResidualStream(x0.clone())
        h = normed(stream, norm_of(w[0], "cuda"), delta, ffn)
        assert isinstance(h, Unnormed) == (shift == 0)
        y = ffn.forward(h)
        assert torch.equal(stream.x, x0 + delta0.float())
        results.append(y.double())
    assert float((results[0] - results[1]).norm() / results[0].norm()) < 2e-2
