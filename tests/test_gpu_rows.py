"""Row kernels around the sizes their launches choose by: cross-entropy rows of few and many vectors per thread, norm
backward with fewer rows than CTAs, several rows per CTA and each register layout, against 64-bit results."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,V", [(1, 8), (5, 4096), (3, 4104), (130, 32000), (7, 32768), (7, 32776)])
def test_linear_cross_entropy_rows(native, N, V):
    torch.manual_seed(V)
    d = 64
    h = (torch.randn(N, d, device="cuda") * 2).bfloat16().requires_grad_()
    w = (torch.randn(V, d, device="cuda") * 0.2).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (N,), device="cuda")
    if N > 4:
        labels[3] = -100
    loss = native.linear_cross_entropy(h, w, labels)
    got = torch.autograd.grad(loss * 3.0, [h, w])
    hr, wr = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    ref = F.cross_entropy(hr @ wr.t(), labels, ignore_index=-100)
    want = torch.autograd.grad(ref * 3.0, [hr, wr])
    assert abs(float(loss) - float(ref)) <= 2e-3 * abs(float(ref)) + 2e-3          # logits are rounded to bf16
    for a, b in zip(got, want):
        assert a.dtype == torch.bfloat16 and (a.double() - b).norm() <= 1.5e-2 * b.norm()


def test_cross_entropy_of_short_rows_costs_little(native):
    # 16384 rows of 512 logits against as many of 32000: 0.09 of the time; 0.33 with CTAs sized for the long rows
    from ctypes import c_int, c_long, c_void_p
    p = lambda t: c_void_p(t.data_ptr())                                            # noqa: E731
    rows = 16384
    labels, losses, inv = torch.zeros(rows, device="cuda", dtype=torch.long), torch.empty(rows, device="cuda"), torch.ones(1, device="cuda")

    def fastest(V):
        logits = torch.randn(rows, V, device="cuda", dtype=torch.bfloat16)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            native._check(native.load().nsa_cross_entropy(p(logits), p(labels), p(losses), p(inv), c_long(rows), c_int(V), c_long(V),
                                                          c_long(-100), c_int(1), native._stream()))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    assert fastest(512) <= 0.2 * fastest(32000)


def test_linear_cross_entropy_gradient_of_the_upstream_factor(native):
    torch.manual_seed(0)
    h = torch.randn(40, 64, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(512, 64, device="cuda") * 0.2).bfloat16().requires_grad_()
    labels = torch.randint(0, 512, (40,), device="cuda")
    loss = native.linear_cross_entropy(h, w, labels)
    plain = torch.autograd.grad(loss, [h, w], retain_graph=True)
    # a batch of factors
    factors = torch.tensor([1.0, -2.0, 0.5], device="cuda")
    many = torch.autograd.grad(loss, [h, w], factors, is_grads_batched=True, retain_graph=True)
    for m, g in zip(many, plain):
        assert m.dtype == g.dtype and torch.equal(m, torch.stack([g, -2.0 * g, 0.5 * g]))     # powers of two: exact
    # the gradient is linear in the factor, and its derivative with respect to the factor is the plain gradient
    a = torch.tensor(1.0, device="cuda", requires_grad=True)
    got = torch.autograd.grad(loss * a, [h, w], create_graph=True)
    for g, ref in zip(got, plain):
        assert torch.equal(g, ref)
        c = torch.randn_like(ref, dtype=torch.float32)
        slope, = torch.autograd.grad((g.float() * c).sum(), a, retain_graph=True)
        want = (ref.float() * c).sum()
        # bf16 products (dh) enter the sum: one rounding of 2^-9 per term at most
        assert abs(float(slope - want)) <= 2 ** -8 * float((ref.float() * c).abs().sum())


@pytest.mark.parametrize("mode", ["plain", "add", "before", "after"])
@pytest.mark.parametrize("rows,d", [(1, 256), (7, 512), (3000, 256), (6000, 264), (1, 2048), (593, 2048), (1300, 1000), (700, 4096), (600, 8192)])
def test_norm_backward_rows(native, mode, rows, d):
    torch.manual_seed(d)
    x, r, dy, dh = (torch.randn(rows, d, device="cuda").bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16()
    leaves = [t.requires_grad_() for t in ([x, w] if mode == "plain" else [x, r, w])]
    ref = [t.detach().double().requires_grad_() for t in leaves]
    norm = lambda u, v: u * (u.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * v     # noqa: E731
    if mode == "add":
        h, y = native.add_rms_norm(*leaves)
        got = torch.autograd.grad([h, y], leaves, [dh, dy])
        # the kernel's statistics are those of the rounded sum
        s = ref[0] + ref[1]
        s = s + (s.to(torch.bfloat16).double() - s).detach()
        want = torch.autograd.grad([s, norm(s, ref[2])], ref, [dh.double(), dy.double()])
    elif mode == "plain":
        got = torch.autograd.grad(native.rms_norm(*leaves), leaves, dy)
        want = torch.autograd.grad(norm(*ref), ref, dy.double())
    else:
        got = torch.autograd.grad(native.gated_rms_norm(*leaves, norm_before_gate=mode == "before"), leaves, dy)
        y = norm(ref[0], ref[2]) * F.silu(ref[1]) if mode == "before" else norm(ref[0] * F.silu(ref[1]), ref[2])
        want = torch.autograd.grad(y, ref, dy.double())
    for a, b in zip(got, want):
        assert (a.double() - b).norm() <= 5e-3 * b.norm() + 1e-6                      # one rounding to bf16, fp32 inside


@pytest.mark.parametrize("mode", ["before", "after"])
@pytest.mark.parametrize("rows,d,pitch", [(3000, 128, 136), (1200, 512, 1024), (900, 4096, 8512), (500, 8192, 8200)])
def test_gated_norm_backward_pitched_gate(native, mode, rows, d, pitch):
    torch.manual_seed(pitch)
    x, dy = (torch.randn(rows, d, device="cuda").bfloat16() for _ in range(2))
    gate = torch.randn(rows, pitch, device="cuda").bfloat16()[:, pitch - d:]
    w = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16()
    leaves = [x.requires_grad_(), gate.requires_grad_(), w.requires_grad_()]
    ref = [t.detach().double().requires_grad_() for t in leaves]
    norm = lambda u, v: u * (u.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * v     # noqa: E731
    got = torch.autograd.grad(native.gated_rms_norm(*leaves, norm_before_gate=mode == "before"), leaves, dy)
    y = norm(ref[0], ref[2]) * F.silu(ref[1]) if mode == "before" else norm(ref[0] * F.silu(ref[1]), ref[2])
    for a, b in zip(got, torch.autograd.grad(y, ref, dy.double())):
        assert (a.double() - b).norm() <= 5e-3 * b.norm() + 1e-6                      # one rounding to bf16, fp32 inside


# 2.1 times the copy at 128 columns with four CTAs per SM, 4.1 with two; 1.2 at 4096 columns with 512 threads a row, 2.2 with 256
@pytest.mark.parametrize("rows,d,limit", [(1 << 20, 128, 3.1), (1 << 16, 4096, 1.7)])
def test_norm_backward_of_many_rows_is_memory_bound(native, rows, d, limit):
    # Three tensors pass through memory; a copy of as many bytes is the yardstick
    x, dy = (torch.randn(rows, d, device="cuda").bfloat16().requires_grad_(i == 0) for i in range(2))
    w = torch.ones(d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = native.rms_norm(x, w)
    src, dst = (torch.empty(rows * d * 3 // 2, device="cuda", dtype=torch.bfloat16) for _ in range(2))

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
    assert fastest(lambda: torch.autograd.grad(y, [x, w], dy, retain_graph=True)) <= limit * copy


def test_a_single_row_of_any_pitch(native):
    # one token of a wider row, which counts as dense: its stride is no pitch that the kernels could take
    g = torch.Generator("cuda").manual_seed(0)
    cut = lambda h, n: torch.randn(1, 5, h * n + 1, device="cuda", generator=g).bfloat16()[..., :h * n].view(1, 5, h, n)[:, :1]      # noqa: E731
    x, Bm, Cm, gate = cut(3, 64), cut(1, 128), cut(1, 128), cut(1, 256)[:, :, 0][0]
    w = torch.rand(256, device="cuda", generator=g).bfloat16()
    dt, A, D = torch.rand(1, 1, 3, device="cuda"), -torch.rand(3, device="cuda"), torch.rand(3, device="cuda")
    assert all(t.is_contiguous() and t.stride(t.dim() // 4) % 8 for t in (x, Bm, Cm, gate))
    for op, inputs in ((native.ssd_scan, (x, dt, A, Bm, Cm, D)), (native.gated_rms_norm, (gate, gate, w)), (native.gated_rms_norm, (gate, gate, w, 1e-6, False))):
        results = []
        for dense in (False, True):
            leaves = [(t.clone(memory_format=torch.contiguous_format) if dense else t).detach().requires_grad_() if isinstance(t, torch.Tensor) else t for t in inputs]
            y = op(*leaves)
            results.append([y.detach(), *torch.autograd.grad(y, [t for t in leaves if isinstance(t, torch.Tensor)], torch.ones_like(y))])
        assert all(torch.equal(a, b) for a, b in zip(*results))
