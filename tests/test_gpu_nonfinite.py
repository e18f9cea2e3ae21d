"""Infinities and NaN stay where the arithmetic puts them: other rows, heads, channels and blocks are untouched, to the bit."""
import pytest
import torch

from nsa_optim_b200.ops import oracle

pytestmark = pytest.mark.gpu
BAD = [float("nan"), float("inf"), float("-inf")]


@pytest.mark.parametrize("mode", ["plain", "add", "before", "after"])
@pytest.mark.parametrize("d", [128, 512, 2048, 4096, 8192])
def test_norm_backward_rows(native, mode, d):
    torch.manual_seed(d)
    rows, bad = 1500, [0, 7, 1499]
    x, r, dy, dh = (torch.randn(rows, d, device="cuda").bfloat16() for _ in range(4))
    w = torch.ones(d, device="cuda", dtype=torch.bfloat16)

    def grads(x):
        leaves = [t.detach().requires_grad_() for t in ([x, w] if mode == "plain" else [x, r, w])]
        if mode == "add":
            return torch.autograd.grad(list(native.add_rms_norm(*leaves)), leaves, [dh, dy])[:-1]
        y = native.rms_norm(*leaves) if mode == "plain" else native.gated_rms_norm(*leaves, norm_before_gate=mode == "before")
        return torch.autograd.grad(y, leaves, dy)[:-1]

    clean = grads(x)
    y = x.clone()
    y[bad, [3, d // 2, d - 1]] = torch.tensor(BAD, device="cuda", dtype=torch.bfloat16)
    keep = [i for i in range(rows) if i not in bad]
    for a, b in zip(clean, grads(y)):
        assert torch.equal(a[keep], b[keep]) and not torch.isfinite(b[bad[0]]).all()


@pytest.mark.parametrize("V", [64, 4096, 32000, 32776])
def test_cross_entropy_rows(native, V):
    from ctypes import c_int, c_long, c_void_p
    p = lambda t: c_void_p(t.data_ptr())                                            # noqa: E731
    torch.manual_seed(V)
    rows = 9
    logits = torch.randn(rows, V, device="cuda").bfloat16()
    labels = torch.randint(0, V, (rows,), device="cuda")
    masked = torch.rand(V, device="cuda") < 0.5                                       # a row with half its words masked out
    masked[::8] = False
    masked[labels[4]] = False
    logits[4, masked] = float("-inf")
    ref = torch.nn.functional.cross_entropy(logits.double(), labels, reduction="none")
    logits[0, 1], logits[2, V - 1] = BAD[0], BAD[1]
    losses, inv = torch.empty(rows, device="cuda"), torch.ones(1, device="cuda")
    native._check(native.load().nsa_cross_entropy(p(logits), p(labels), p(losses), p(inv), c_long(rows), c_int(V), c_long(V),
                                                  c_long(-100), c_int(1), native._stream()))
    good = [1, 3, 4, 5, 6, 7, 8]
    assert torch.isfinite(logits[good]).all() and not torch.isfinite(losses[[0, 2]]).any()
    assert (losses[good].double() - ref[good]).abs().max() <= 1e-4 * ref.max()       # fp32 sums of bf16 logits
    assert (logits[4, masked] == 0).all()


def test_adamw8bit_blocks(native):
    torch.manual_seed(0)
    n = 256 * 40

    def update(g):
        torch.manual_seed(1)
        state = [torch.randn(n, device="cuda"), torch.randint(0, 256, (n,), device="cuda").to(torch.uint8), torch.rand(n // 256, device="cuda"),
                 torch.randint(128, 256, (n,), device="cuda").to(torch.uint8), torch.rand(n // 256, device="cuda")]
        native.adamw8bit_step(state[0], g, *state[1:], 3, 1e-3, 0.9, 0.95, 1e-8, 0.1, None, 256)
        return [t.view(40, -1) for t in state]

    g = torch.randn(n, device="cuda")
    clean = update(g)
    g[[5, 256 * 11 + 200, 256 * 39]] = torch.tensor(BAD, device="cuda")
    keep = [b for b in range(40) if b not in (0, 11, 39)]
    for a, b in zip(clean, update(g)):
        assert torch.equal(a[keep], b[keep])


def test_conv1d_channels_and_steps(native):
    torch.manual_seed(0)
    x, dy = (torch.randn(2, 300, 136, device="cuda").bfloat16() for _ in range(2))
    w, b = torch.randn(136, 4, device="cuda").bfloat16(), torch.randn(136, device="cuda").bfloat16()

    def run(x):
        leaves = [t.detach().requires_grad_() for t in (x, w, b)]
        y = native.causal_conv1d(*leaves)
        return [y.detach()] + list(torch.autograd.grad(y, leaves, dy))

    clean, z = run(x), x.clone()
    z[1, 100, 5], z[0, 299, 135] = BAD[0], BAD[1]
    got = run(z)
    touched = torch.zeros(2, 300, 136, dtype=torch.bool, device="cuda")
    touched[1, 97:104, 5] = True                                                      # the taps that see step 100, either way
    touched[0, 296:, 135] = True
    for a, b_ in zip(clean[:2], got[:2]):
        assert torch.equal(a[~touched], b_[~touched]) and not torch.isfinite(b_[touched]).all()
    others = [c for c in range(136) if c not in (5, 135)]
    assert all(torch.equal(a[others], b_[others]) for a, b_ in zip(clean[2:], got[2:]))


@pytest.mark.parametrize("value", BAD[:2])
def test_heads_of_the_scans(native, value):
    torch.manual_seed(0)
    B, T, H = 1, 300, 4
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()                       # noqa: E731
    unit = lambda t: oracle.l2_norm(t.float()).bfloat16()                            # noqa: E731
    gate, beta = -torch.rand(B, T, H, device="cuda"), torch.rand(B, T, H, device="cuda")
    delta = [unit(rnd(B, T, H, 128)), unit(rnd(B, T, H, 128)), rnd(B, T, H, 128), gate, beta]
    scan = [rnd(B, T, H, 64), beta, -torch.rand(H, device="cuda") - 1, rnd(B, T, 1, 128), rnd(B, T, 1, 128), torch.ones(H, device="cuda")]
    for op, inputs, where, kept in ((native.gated_delta_rule, delta, 2, 5), (native.ssd_scan, scan, 0, 2)):
        dy = rnd(*inputs[where].shape)

        def run(bad):
            leaves = [t.clone() for t in inputs]
            if bad:
                leaves[where][0, 200, 2, 3] = value
            leaves = [t.requires_grad_() for t in leaves]
            y = op(*leaves)
            return [y.detach()] + list(torch.autograd.grad(y, leaves, dy))[:kept]     # what belongs to a head

        clean, got = run(False), run(True)
        for a, b in zip(clean, got):
            assert torch.equal(a[:, :, [0, 1, 3]], b[:, :, [0, 1, 3]])
        # within the head: the chunks before (64 or 128 tokens) in the output, and what follows is not finite
        assert torch.equal(clean[0][:, :128, 2], got[0][:, :128, 2]) and not torch.isfinite(got[0][:, 200:, 2]).all()
