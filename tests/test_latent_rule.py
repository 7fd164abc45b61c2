"""Which steps of the latent attention part run over expanded latents (no GPU needed)."""
import pytest
import torch


@pytest.mark.parametrize("reqs,wanted", [
    ([(0, 64)], True), ([(0, 600)], True),                                     # prompts alone
    ([(0, 64)] + [(1000, 1)] * 8, False), ([(0, 600)] + [(1000, 1)] * 8, False), ([(2000, 256)] + [(1000, 1)] * 8, False),
    ([(0, 1024)] + [(1000, 1)] * 8, True), ([(1000, 1), (0, 2048)], True), ([(4000, 256)] + [(1000, 1)] * 8, True)])
def test_which_steps_run_over_expanded_latents(reqs, wanted, monkeypatch):
    """The rule at 16 heads of 128 + 64 and a latent of 512, kernel by kernel: where the step was measured to be faster so."""
    from types import SimpleNamespace
    from dinfer_b200.parts import latent_attention as A
    monkeypatch.setattr(A, "num_sms", lambda: 148)
    part = A.LatentAttention.__new__(A.LatentAttention)
    part.H, part.D, part.P, part.V, part.R, part.window, part.ukv = 16, 128, 64, 128, 512, None, object()
    cu = [sum(n for _, n in reqs[:i]) for i in range(len(reqs) + 1)]
    step = dict(cu_seqlens_host=cu, seq_lens_host=[h + n for h, n in reqs], any_decode=any(n == 1 for _, n in reqs), any_prefill=True,
                max_seq_len=max(h + n for h, n in reqs), max_prefill_seq_len=0)
    shape = lambda **kw: part._expanded(SimpleNamespace(**step, derived={}, **kw), torch.bfloat16)
    assert (shape(decode_splits=0) is not None) is wanted
    # without tensor cores for the single tokens there is nothing to gain beside them
    part.P = 40
    assert (shape(decode_splits=0) is not None) is (wanted and not step["any_decode"])
