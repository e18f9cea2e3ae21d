"""Causal convolution over the segment lengths its launch chooses between: sequences shorter than the halo, around
segment ends, and long enough for the longest segments; column counts off the 128-channel tile."""
import pytest
import torch

from nsa_optim_b200.ops import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C", [(1, 1, 8), (2, 2, 136), (1, 3, 120), (3, 7, 128), (1, 63, 256), (2, 64, 8), (1, 65, 1000), (1, 129, 264),
                                   (2, 1023, 1024), (1, 2049, 4096), (1, 9001, 4352), (2, 4608, 4352)])
@pytest.mark.parametrize("act,bias,wdt", [(True, True, torch.bfloat16), (False, False, torch.float32)])
def test_conv1d_segments(native, B, T, C, act, bias, wdt):
    torch.manual_seed(T)
    wide = torch.randn(B, T, C + 16, device="cuda").bfloat16()
    x = wide[..., 8:8 + C].detach().requires_grad_()                              # row pitch wider than C
    w = (torch.randn(C, 4, device="cuda") * 0.4).to(wdt).requires_grad_()
    b = (torch.randn(C, device="cuda") * 0.4).to(wdt).requires_grad_() if bias else None
    dy = torch.randn(B, T, C, device="cuda").bfloat16()
    leaves = [x, w] + ([b] if bias else [])
    y = native.causal_conv1d(x, w, b, act)
    got = [y.detach()] + list(torch.autograd.grad(y, leaves, dy))
    ref = [t.detach().double().requires_grad_() for t in [x, w.to(torch.bfloat16)] + ([b.to(torch.bfloat16)] if bias else [])]
    xp = torch.nn.functional.pad(ref[0], (0, 0, 3, 0))
    yr = sum(xp[:, j:j + T] * ref[1][:, j] for j in range(4)) + (ref[2] if bias else 0)
    yr = torch.nn.functional.silu(yr) if act else yr
    want = [yr.detach()] + list(torch.autograd.grad(yr, ref, dy.double()))
    for a, r in zip(got, want):
        # one rounding to bf16 (2^-9) of values whose fp32 sums are far closer; weight gradients in wdt
        assert a.shape == r.shape and (a.double() - r).norm() <= 3e-3 * r.norm() + 1e-6
        assert (a.double() - r).abs().max() <= 5e-3 * r.abs().max() + 1e-5
    short = oracle.causal_conv1d(x.detach(), w.detach().to(torch.bfloat16), None if b is None else b.detach().to(torch.bfloat16), act)
    assert (got[0].float() - short.float()).abs().max() <= 2 ** -7 * short.float().abs().max() + 1e-5


def test_conv1d_past_65535_segments(native):
    test_conv1d_segments(native, 1, 8388500, 8, True, True, torch.bfloat16)
