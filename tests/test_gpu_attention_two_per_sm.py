"""Forward attention with so many query tiles that two CTAs share an SM: tiles cut off, one visit and many, with and without
causality and window, groups of one head to 32, and selected blocks; a tile more or less on either side of the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(native, q, k, v, seen, got):
    """got against 64 bits; seen (B, Hkv, T, S).  Probabilities and the output are rounded to bf16 (8 bits: 2^-8 each), scores are sums
    of 128 fp32 products of up to |q||k|, exp2 is exact to 2^-22, and up to 2^-13 is left for the fp32 sums over keys."""
    qd, kd, vd = (t.double().transpose(1, 2) for t in (q, k, v))
    G, scale = qd.shape[1] // kd.shape[1], q.shape[-1] ** -0.5
    size = float(qd.norm(dim=-1).max() * kd.norm(dim=-1).max()) * scale
    for h in range(kd.shape[1]):                               # a KV head at a time: the scores in 64 bits are large
        s = (qd[:, h * G:(h + 1) * G] @ kd[:, h, None].transpose(-1, -2) * scale).masked_fill(~seen[:, h, None], -float("inf"))
        p = s.softmax(-1).nan_to_num(0.0)
        want, mass = p @ vd[:, h, None], p @ vd[:, h, None].abs()
        err = (got.double().transpose(1, 2)[:, h * G:(h + 1) * G] - want).abs()
        bound = 2.0 ** -8 * want.abs() + (2.0 ** -8 + 2.0 ** -13 + 2.0 ** -24 * 130 * size) * mass
        assert (err <= 1.01 * bound + 1e-6).all(), float((err / (bound + 1e-9)).max())


@pytest.mark.parametrize("B,T,Hq,Hkv,causal,window", [
    (1, 1184, 32, 2, True, 0), (1, 1176, 32, 2, True, 0),      # 296 and 294 tiles of up to 19 visits
    (4, 1191, 16, 2, False, 0), (2, 1500, 32, 2, True, 100), (40, 33, 16, 8, True, 0), (300, 1, 2, 1, True, 0), (19, 130, 16, 16, False, 64),
    (1, 1200, 32, 1, True, 0),                                 # groups of 32: 300 tiles of 4 tokens
    (2, 1340, 32, 2, True, 700), (1, 2400, 32, 2, False, 0),   # more than 20 visits
    (8, 1400, 16, 8, True, 0)])
def test_forward(native, B, T, Hq, Hkv, causal, window):
    g = torch.Generator("cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, h, 128, device="cuda", generator=g).bfloat16() for h in (Hq, Hkv, Hkv))
    t = torch.arange(T, device="cuda")
    seen = (t[None, :] <= t[:, None]) if causal else torch.ones(T, T, dtype=torch.bool, device="cuda")
    if window:
        seen = seen & (t[None, :] > t[:, None] - window)
    _check(native, q, k, v, seen.expand(B, Hkv, T, T), native.attention(q, k, v, causal, window))


@pytest.mark.parametrize("T,Hq,Hkv", [(1184, 32, 2), (2380, 32, 2)])
def test_selected(native, T, Hq, Hkv):
    g = torch.Generator("cuda").manual_seed(T)
    q, k, v = (torch.randn(1, T, h, 128, device="cuda", generator=g).bfloat16() for h in (Hq, Hkv, Hkv))
    nS, t = -(-T // 64), torch.arange(T, device="cuda")
    own = (t // 64)[None, None, :, None]
    pick = torch.randint(0, nS, (1, Hkv, T, 4), device="cuda", generator=g)
    idx = torch.cat([own.expand(1, Hkv, T, 1), torch.where(pick <= own, pick, -1)], -1).to(torch.int32)
    took = torch.zeros(1, Hkv, T, nS + 1, dtype=torch.bool, device="cuda").scatter_(-1, torch.where(idx < 0, nS, idx).long(), True)
    seen = took[..., :nS].repeat_interleave(64, -1)[..., :T] & (t[None, :] <= t[:, None])
    _check(native, q, k, v, seen, native.selected_attention(q, k, v, idx))
