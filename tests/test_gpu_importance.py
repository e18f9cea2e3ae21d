"""Block importance at the group sizes and lengths where its sum over heads, its bins and its tiles have edges: probabilities of
the compressed keys, summed over the heads of a group, each key into the blocks of its two cells."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 2, 8, 16, 32])
@pytest.mark.parametrize("T", [31, 32, 1055, 1056, 2063])     # no key, one, 64 and 65 (a second visit), the last block cut off
def test_importance_against_64_bits(native, G, T):
    B, Hkv, D, stride, block = 2, 2, 128, 16, 32
    S, nS, scale = max(1, (T - block) // stride + 1), (T + 63) // 64, 128 ** -0.5
    torch.manual_seed(G * 7 + T)
    q = torch.randn(B, T, Hkv * G, D, device="cuda").bfloat16()
    k = torch.randn(B, S, Hkv, D, device="cuda").bfloat16()
    qd, kd = q.double().view(B, T, Hkv, G, D), k.double()
    seen = torch.arange(S, device="cuda")[None] * stride + block - 1 <= torch.arange(T, device="cuda")[:, None]
    s = torch.einsum("bthgd,bshd->bhgts", qd, kd).mul(scale / math.log(2)).masked_fill(~seen, -math.inf)
    L = (torch.logsumexp(s * math.log(2), -1) / math.log(2)).float()                     # (B, Hkv, G, T), base 2
    p = torch.where(seen, torch.exp2(s - L.double().nan_to_num(neginf=0)[..., None]), 0.0).sum(2)
    want = torch.zeros(B, Hkv, T, nS + 1, dtype=torch.double, device="cuda")
    i = torch.arange(S, device="cuda")
    for cell in (i, i + 1):
        want.index_add_(3, cell // 4, p)
    want = want[..., :nS]
    got = native.nsa_importance(q, k, L.permute(0, 3, 1, 2).reshape(B, T, Hkv * G).contiguous(), nS, stride, block, scale)
    # relative error of a probability: D fp32 additions of products of at most max |q||k| each, the exponent's own rounding, exp2 to
    # 2^-22; then up to 8 G additions per bin
    size = float(qd.norm(dim=-1).max() * kd.norm(dim=-1).max()) * scale
    bound = 2.0 ** -24 * ((D + 2) * size + 4 * float(L.abs().nan_to_num(posinf=0).max()) + 8 * G) + 2.0 ** -21
    assert ((got.double() - want).abs() <= bound * want + 1e-30).all()
