"""Attention of head_dim 64, forward and backward: tiles and key blocks that the sequence ends inside, one visit and many, groups of one head to
64, windows, without causality, one walk of a key block and several; selected blocks; twice the same bits where the sums are ordered."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, seen):
    """64 bits; seen (B, Hkv, T, S)."""
    q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    G = q.shape[1] // k.shape[1]
    k, v, seen = (t.repeat_interleave(G, 1) for t in (k, v, seen))
    p = (q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5).masked_fill(~seen, -float("inf")).softmax(-1).nan_to_num(0.0)
    return (p @ v).transpose(1, 2)


def _range(T, window, causal):
    t = torch.arange(T, device="cuda")
    seen = t[None, :] <= t[:, None] if causal else torch.ones(T, T, dtype=torch.bool, device="cuda")
    return seen & (t[None, :] > t[:, None] - window) if window else seen


def _check(native, B, T, Hq, Hkv, window, causal):
    g = torch.Generator("cuda").manual_seed(T)
    mk = lambda h: torch.randn(B, T, h, 64, device="cuda", generator=g).bfloat16().requires_grad_()      # noqa: E731
    x, dy = [mk(Hq), mk(Hkv), mk(Hkv)], mk(Hq).detach()

    def run():
        y = native.attention(*x, causal, window)
        return [y.detach()] + list(torch.autograd.grad(y, x, dy))

    got, again = run(), run()
    ref = [t.detach().double().requires_grad_() for t in x]
    y = _reference(*ref, _range(T, window, causal).expand(B, Hkv, T, T))
    want = [y.detach()] + list(torch.autograd.grad(y, ref, dy.double()))
    native.check_status()
    for a, b, w in zip(got, again, want):
        # probabilities, score gradients and the result are rounded to bf16: 2^-8 at most, 2^-9 in the mean.  A token that sees one key has score gradients
        # of zero, as the difference of two fp32 sums of 64 products of size one: 64 * 2^-24 per element at most
        assert (a.double() - w).norm() <= 3 * 2 ** -9 * w.norm() + 2 ** -18 * a.numel() ** 0.5
        if T * Hq // Hkv <= 256 * 128:               # up to 256 query tiles: every sum in a fixed order
            assert torch.equal(a, b)


@pytest.mark.parametrize("B,T,Hq,Hkv,window", [
    (1, 1, 4, 4, 0), (2, 17, 2, 2, 5), (1, 128, 64, 1, 0), (1, 129, 16, 2, 0), (2, 300, 16, 8, 0), (1, 640, 32, 2, 127), (1, 900, 32, 1, 129),
    (1, 700, 8, 8, 300), (4, 777, 16, 8, 512), (1, 2100, 32, 1, 0), (40, 33, 16, 8, 0), (19, 130, 16, 16, 64), (2, 1500, 16, 16, 0),
    (1, 592, 32, 2, 0), (1, 600, 32, 2, 0), (1, 1768, 32, 2, 0), (1, 1776, 32, 2, 0)])    # 148, 150, 442 and 444 tiles: one CTA per SM and two
def test_causal(native, B, T, Hq, Hkv, window):
    _check(native, B, T, Hq, Hkv, window, True)


@pytest.mark.parametrize("window", [0, 64, 512])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 300, 16, 1), (4, 600, 16, 16), (1, 769, 16, 1), (1, 1100, 32, 1)])
def test_without_causality(native, B, T, Hq, Hkv, window):
    _check(native, B, T, Hq, Hkv, window, False)


@pytest.mark.parametrize("walks", [1, 2, 5, 64])
@pytest.mark.parametrize("B,T,Hq,Hkv,window,causal", [(1, 1, 4, 4, 0, True), (2, 65, 8, 1, 0, True), (1, 300, 16, 8, 64, False), (1, 520, 32, 2, 129, True),
                                                      (2, 333, 16, 2, 0, False)])
def test_walks(native, monkeypatch, B, T, Hq, Hkv, window, causal, walks):
    monkeypatch.setattr(native.load(), "nsa_attn_bwd_walks_d64", lambda *args: walks)
    _check(native, B, T, Hq, Hkv, window, causal)


@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 300, 4, 2), (2, 1184, 32, 2), (1, 64, 16, 1)])
def test_selected(native, B, T, Hq, Hkv):
    g = torch.Generator("cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, h, 64, device="cuda", generator=g).bfloat16() for h in (Hq, Hkv, Hkv))
    nS, t = -(-T // 64), torch.arange(T, device="cuda")
    own = (t // 64)[None, None, :, None]
    pick = torch.randint(0, nS, (B, Hkv, T, 4), device="cuda", generator=g)
    idx = torch.cat([own.expand(B, Hkv, T, 1), torch.where(pick <= own, pick, -1)], -1).to(torch.int32)
    took = torch.zeros(B, Hkv, T, nS + 1, dtype=torch.bool, device="cuda").scatter_(-1, torch.where(idx < 0, nS, idx).long(), True)
    seen = took[..., :nS].repeat_interleave(64, -1)[..., :T] & (t[None, :] <= t[:, None])
    got, want = native.selected_attention(q, k, v, idx).double(), _reference(q.double(), k.double(), v.double(), seen)
    assert (got - want).norm() <= 3 * 2 ** -9 * want.norm()


# Keys of 32 tokens every 16: the first 31 tokens see none (L = -inf).  32 tokens have one key; a group of 32 heads over 2100 tokens has more than 256
# query tiles, whose sums meet in memory
@pytest.mark.parametrize("walks", [None, 1, 3])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 32, 4, 2), (2, 300, 16, 8), (1, 1000, 16, 1), (1, 2080, 8, 4), (1, 2100, 32, 1)])
def test_compressed_keys(native, monkeypatch, B, T, Hq, Hkv, walks):
    if walks:
        monkeypatch.setattr(native.load(), "nsa_attn_bwd_walks_d64", lambda *args: walks)
    g = torch.Generator("cuda").manual_seed(T)
    S = (T - 32) // 16 + 1
    mk = lambda t, h: torch.randn(B, t, h, 64, device="cuda", generator=g).bfloat16().requires_grad_()      # noqa: E731
    x, dy = [mk(T, Hq), mk(S, Hkv), mk(S, Hkv)], mk(T, Hq).detach()
    seen = torch.arange(S, device="cuda")[None, :] * 16 + 31 <= torch.arange(T, device="cuda")[:, None]
    y, L = native._Attn.apply(*x, True, 0, 0.125, 16, 31, None)
    got = [y.detach()] + list(torch.autograd.grad(y, x, dy))
    ref = [t.detach().double().requires_grad_() for t in x]
    # unseen keys at -1e30 and not -inf, whose softmax over nothing has no gradient; its result is taken out afterwards
    G = Hq // Hkv
    q, k, v = ref[0].transpose(1, 2), *(t.transpose(1, 2).repeat_interleave(G, 1) for t in ref[1:])
    s = (q @ k.transpose(-1, -2) * 0.125).masked_fill(~seen, -1e30)
    w = ((s.softmax(-1) * seen) @ v).transpose(1, 2)
    want = [w.detach()] + list(torch.autograd.grad(w, ref, dy.double()))
    native.check_status()
    assert torch.isneginf(L[:, :31]).all() and torch.isfinite(L[:, 31:]).all()
    assert not y[:, :31].any() and not got[1][:, :31].any()
    for a, b in zip(got, want):                    # as in _check; S = 1: score gradients are differences of equal sums
        assert (a.double() - b).norm() <= 3 * 2 ** -9 * b.norm() + 2 ** -18 * a.numel() ** 0.5
