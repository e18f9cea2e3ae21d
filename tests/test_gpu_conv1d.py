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
    # both ends against runs over the ends alone, the weight gradient against sums of pieces in 64 bits
    torch.manual_seed(0)
    T, C, n = 8388500, 264, 1000
    x, dy = (torch.randn(1, T, C, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    w = (torch.randn(C, 4, device="cuda") * 0.4).requires_grad_()

    def run(part):
        xs = x[:, part].detach().requires_grad_()
        y = native.causal_conv1d(xs, w, None, False)
        return [y.detach()] + list(torch.autograd.grad(y, [xs, w], dy[:, part]))

    y, dx, dw = run(slice(0, T))
    ys, dxs, _ = run(slice(0, n + 3))
    assert torch.equal(y[:, :n], ys[:, :n]) and torch.equal(dx[:, :n], dxs[:, :n])
    ys, dxs, _ = run(slice(T - n, T))
    assert torch.equal(y[:, T - n + 3:], ys[:, 3:]) and torch.equal(dx[:, T - n:], dxs)
    want = torch.zeros(C, 4, device="cuda", dtype=torch.float64)
    for s in range(0, T, 1 << 18):
        e = min(T, s + (1 << 18))
        xs = torch.nn.functional.pad(x[0, max(0, s - 3):e].double(), (0, 0, 3 - min(s, 3), 0))
        want += torch.stack([(dy[0, s:e].double() * xs[j:j + e - s]).sum(0) for j in range(4)], 1)
    assert (dw.double() - want).norm() <= 1e-5 * T ** 0.5 * want.numel() ** 0.5    # sums of T products of size one, in fp32


def test_conv1d_backward_of_few_channels_fills_the_sms(native):
    # 128 channels are one tile: all eight warps of a CTA take time segments.  A copy of as many bytes is the yardstick
    T, C = 1 << 19, 128
    x, dy = (torch.randn(1, T, C, device="cuda").bfloat16().requires_grad_(i == 0) for i in range(2))
    w = torch.randn(C, 4, device="cuda").bfloat16().requires_grad_()
    y = native.causal_conv1d(x, w, None, True)
    src, dst = (torch.empty(3 * T * C // 2, device="cuda", dtype=torch.bfloat16) for _ in range(2))

    def fastest(call):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    copy = fastest(lambda: dst.copy_(src))
    back = fastest(lambda: torch.autograd.grad(y, [x, w], dy, retain_graph=True))
    assert back <= 4.5 * copy, (back, copy)
