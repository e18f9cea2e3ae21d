"""dK / dV over contiguous key ranges: blocks of 64 and of 128 keys that the sequence ends inside, groups from one head to 32, windows around a
block's length, one walk a block and several, and several sequences; twice the same bits where the sums are ordered."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, window, causal=True):
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    G, T = q.shape[1] // k.shape[1], q.shape[2]
    k, v = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)
    t = torch.arange(T, device=q.device)
    seen = t[None, :] <= t[:, None] if causal else torch.ones(T, T, dtype=torch.bool, device=q.device)
    if window:
        seen &= t[None, :] > t[:, None] - window
    p = (q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5).masked_fill(~seen, -float("inf")).softmax(-1)
    return (p @ v).transpose(1, 2)


def _check(native, B, T, Hq, Hkv, window, causal):
    g = torch.Generator("cuda").manual_seed(T)
    mk = lambda h: torch.randn(B, T, h, 128, device="cuda", generator=g).bfloat16().requires_grad_()      # noqa: E731
    x, dy = [mk(Hq), mk(Hkv), mk(Hkv)], mk(Hq).detach()
    run = lambda: torch.autograd.grad(native.attention(*x, causal, window), x, dy)                        # noqa: E731
    got, again = run(), run()
    ref = [t.detach().double().requires_grad_() for t in x]
    want = torch.autograd.grad(_reference(*ref, window, causal), ref, dy.double())
    native.check_status()
    for a, b, w in zip(got, again, want):
        # probabilities, score gradients and the result are rounded to bf16: 2^-8 at most, 2^-9 in the mean.  A token that sees one key has score gradients
        # of zero, as the difference of two fp32 sums of 128 products of size one: 128 * 2^-24 per element at most
        assert (a.double() - w).norm() <= 3 * 2 ** -9 * w.norm() + 2 ** -17 * a.numel() ** 0.5
        if T * Hq // Hkv <= 256 * 128:               # up to 256 query tiles: every sum in a fixed order
            assert torch.equal(a, b)


@pytest.mark.parametrize("B,T,Hq,Hkv,window", [(1, 1, 4, 4, 0), (2, 17, 2, 2, 5), (1, 128, 32, 1, 0), (1, 129, 16, 2, 0), (2, 300, 16, 8, 0),
                                               (1, 640, 32, 2, 127), (1, 900, 32, 1, 129), (1, 700, 8, 8, 300), (1, 2100, 32, 1, 0)])
def test_key_gradients(native, B, T, Hq, Hkv, window):
    _check(native, B, T, Hq, Hkv, window, True)


# Without causality a key is seen by every token up to a window after it, so the last key blocks have all query tiles: one walk
# a block and several, and (32 heads a group, 1100 tokens) more than 256 tiles
@pytest.mark.parametrize("window", [0, 64, 512])
@pytest.mark.parametrize("T,Hq,Hkv", [(300, 16, 1), (600, 4, 4), (600, 8, 4), (769, 16, 1), (1000, 2, 1), (1000, 16, 1), (1025, 8, 8),
                                      (1100, 32, 1)])
def test_key_gradients_without_causality(native, T, Hq, Hkv, window):
    _check(native, 1, T, Hq, Hkv, window, False)


# "No limit" written as a number: positions plus the window pass 2^31.  Several walks a block, and more than 256 tiles
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("T,Hq,Hkv,window", [(300, 16, 1, 2 ** 31 - 1), (300, 2, 2, 2 ** 31 - 129), (1100, 32, 1, 2 ** 31 - 1), (300, 16, 1, 300)])
def test_key_gradients_of_the_widest_windows(native, T, Hq, Hkv, window, causal):
    _check(native, 1, T, Hq, Hkv, window, causal)


# Every form on ranges that the rule may give to another: 64 keys a CTA, one walk of 128 keys, several, one visit each
@pytest.mark.parametrize("form", [-1, 1, 2, 5, 64])
@pytest.mark.parametrize("B,T,Hq,Hkv,window,causal", [(1, 1, 4, 4, 0, True), (2, 65, 8, 1, 0, True), (1, 127, 16, 16, 0, True), (1, 300, 16, 8, 64, True),
                                                      (1, 300, 16, 8, 64, False), (1, 520, 32, 2, 129, True), (2, 333, 16, 2, 0, False)])
def test_forms(native, monkeypatch, B, T, Hq, Hkv, window, causal, form):
    monkeypatch.setattr(native.load(), "nsa_attn_bwd_walks", lambda *args: form)
    _check(native, B, T, Hq, Hkv, window, causal)


# Where few tiles visit a block the smaller blocks are faster, also with a window, and where blocks are few several walks are.  us
# (64 keys; 128 keys and one walk; and several): 7.4, 10; 12.9, 17; 9.5, 14.4; 20, 32, 24; 181, 210, 33; 51, 46, 56
@pytest.mark.parametrize("T,Hq,Hkv,window,low,high", [(128, 16, 16, 0, -1, -1), (300, 16, 8, 0, -1, -1), (1000, 16, 8, 64, -1, -1),
                                                      (3000, 16, 2, 64, -1, -1), (1000, 32, 2, 0, 12, 20), (1500, 16, 16, 0, 1, 1)])
def test_choice_of_form(native, T, Hq, Hkv, window, low, high):
    assert low <= native.load().nsa_attn_bwd_walks(1, T, T, Hq, Hkv, 1, window, 1) <= high
