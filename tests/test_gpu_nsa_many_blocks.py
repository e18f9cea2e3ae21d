"""Native sparse attention with more selected blocks per token than the kernels that invert a selection take: forward and gradients of the one
node against plain attention in 64 bits over the same blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _attend(q, k, v, seen):
    """q (B, T, Hq, D), k, v (B, S, Hkv, D), seen (B, Hkv or 1, T, S); tokens that see nothing get zero."""
    G = q.shape[2] // k.shape[2]
    q, k, v = q.transpose(1, 2), *(t.transpose(1, 2).repeat_interleave(G, 1) for t in (k, v))
    seen = seen.expand(-1, k.shape[1] // G, -1, -1).repeat_interleave(G, 1)
    s = (q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5).masked_fill(~seen, -1e30)
    return ((s.softmax(-1) * seen) @ v).transpose(1, 2)


def _plain(q, k, v, gates, idx, window):
    B, T, Hq, _ = q.shape
    pool = lambda x: x.unfold(1, 32, 16).mean(-1)                                          # noqa: E731
    kc, vc = pool(k), pool(v)
    t = torch.arange(T, device=q.device)
    causal = t[None, :] <= t[:, None]
    took = torch.zeros(*idx.shape[:3], -(-T // 64) + 1, dtype=torch.bool, device=q.device)
    took.scatter_(-1, torch.where(idx < 0, took.shape[-1] - 1, idx).long(), True)
    seen = (torch.arange(kc.shape[1], device=q.device)[None, :] * 16 + 31 <= t[:, None],
            took[..., :-1].repeat_interleave(64, -1)[..., :T] & causal,
            causal & (t[None, :] > t[:, None] - window))
    o = [_attend(q, a, b, m if m.dim() == 4 else m[None, None]) for a, b, m in zip((kc, k, k), (vc, v, v), seen)]
    return sum(g[..., None] * x for g, x in zip(torch.sigmoid(gates).split(Hq, -1), o))


# 33 entries are one more than the kernels take; 48 are more than there are blocks, so that every visible one is selected
@pytest.mark.parametrize("B,T,Hq,Hkv,top_n", [(1, 2300, 8, 1, 33), (2, 2240, 16, 2, 34), (1, 1000, 16, 1, 48)])
def test_more_than_32_selected_blocks(native, B, T, Hq, Hkv, top_n):
    g = torch.Generator("cuda").manual_seed(T)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16().requires_grad_()   # noqa: E731
    x, dy = [mk(B, T, Hq, 128), mk(B, T, Hkv, 128), mk(B, T, Hkv, 128), mk(B, T, 3 * Hq)], mk(B, T, Hq, 128).detach()
    y = native.nsa_attention(*x[:3], None, None, None, top_n=top_n, window=100, gate_logits=x[3])
    got = [y.detach()] + list(torch.autograd.grad(y, x, dy))
    with torch.no_grad():                                # the blocks that the node chose
        kc = native.nsa_compress(x[1], 32, 16)
        L = native._Attn.apply(x[0], kc, kc, True, 0, 128 ** -0.5, 16, 31, None)[1]
        idx = native.nsa_select(native.nsa_importance(x[0], kc, L, -(-T // 64), 16, 32, 128 ** -0.5), 64, top_n)
    ref = [t.detach().double().requires_grad_() for t in x]
    w = _plain(*ref, idx, 100)
    want = [w.detach()] + list(torch.autograd.grad(w, ref, dy.double()))
    native.check_status()
    for a, b in zip(got, want):
        # pooled keys and values, probabilities, score gradients, a branch's output (or its gradient), partial sums and the result are rounded to
        # bf16 on the way: six times 2^-9 in the mean
        assert (a.double() - b).norm() <= 6 * 2 ** -9 * b.norm()
