"""dK / dV over contiguous key ranges: blocks of 128 keys that the sequence ends inside, groups from one head to 32, windows around a
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
