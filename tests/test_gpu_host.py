"""The ops' host side: guard zones around every output, forward and backward, several threads on streams of their own, and shapes that are
refused before anything is launched."""
import threading

import numpy as np
import pytest
import torch
from test_gpu_unrecorded import _cases

pytestmark = pytest.mark.gpu


def _results(op, inputs):
    leaves = [t.detach().clone().requires_grad_() for t in inputs]
    y = op(*leaves)
    ys = y if isinstance(y, tuple) else (y,)
    return [t.detach() for t in ys] + list(torch.autograd.grad(ys, leaves, [torch.ones_like(t) for t in ys]))


def test_guard_zones_give_the_same_bits(native, monkeypatch):
    cases = _cases(native)
    want = {name: _results(op, inputs) for name, (op, *inputs) in cases.items()}
    monkeypatch.setattr(native, "_CANARY", True)
    for name, (op, *inputs) in cases.items():
        native._guards.clear()
        got = _results(op, inputs)
        assert len(native._guards) >= len(got) and native.check_canaries() > 0, name
        assert all(torch.equal(a, b) for a, b in zip(got, want[name])), name


def test_threads(native):
    cases = _cases(native)
    want = {name: _results(op, inputs) for name, (op, *inputs) in cases.items()}
    torch.cuda.synchronize()
    wrong = []

    def work():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(3):
                for name, (op, *inputs) in cases.items():
                    got = _results(op, inputs)
                    stream.synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, want[name])):
                        wrong.append(name)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_refused_shapes(native):
    r = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)                # noqa: E731
    f = torch.zeros(8, 32, device="cuda")
    for call in (lambda: native.causal_conv1d(r(1, 1, 8, 64), r(64, 4), None), lambda: native.rope(r(1, 8, 2, 1, 64), f, f),
                 lambda: native.linear_cross_entropy(r(1, 8, 64), r(64, 64), torch.zeros(8, device="cuda", dtype=torch.long)),
                 lambda: native.attention(r(1, 8, 2, 64, 1), r(1, 8, 2, 64), r(1, 8, 2, 64)), lambda: native.nsa_compress(r(1, 64, 2, 8, 8), 32, 16),
                 lambda: native.ssd_scan(r(1, 1, 8, 2, 64), f, f, r(1, 8, 1, 128), r(1, 8, 1, 128)),
                 lambda: native.gemm(r(8, 64), r(8, 32), False, False),
                 lambda: native.adamw_multi([(r(8), r(8), f[0, :8], f[0, :4], None, None)], 1, 1e-3, .9, .95, 1e-8, 0.0, None)):
        before = native.launch_count()
        with pytest.raises((ValueError, IndexError, RuntimeError)):
            call()
        assert native.launch_count() == before


def test_chunks_of_the_cross_entropy(native):
    g = torch.Generator("cuda").manual_seed(0)
    h, w = (torch.randn(n, 64, device="cuda", generator=g).bfloat16().requires_grad_() for n in (300, 128))
    ids = torch.randint(0, 128, (300,), device="cuda", generator=g)
    before = native.launch_count()
    for chunk in (0, -1, -2 ** 70):
        with pytest.raises(ValueError):
            native.linear_cross_entropy(h, w, ids, chunk=chunk)
        with pytest.raises(ValueError):
            native.linear_cross_entropy(h[:0], w, ids[:0], chunk=chunk)
    assert native.launch_count() == before
    grads = lambda **kw: torch.autograd.grad(native.linear_cross_entropy(h, w, ids, **kw), (h, w))       # noqa: E731
    for chunk in (300, 2 ** 63 - 1, 2 ** 70):
        assert all(torch.equal(a, b) for a, b in zip(grads(chunk=chunk), grads()))


def test_sizes_of_zero_are_refused(native):
    # each is a divisor on the host: an exception, not the end of the process
    r = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)                # noqa: E731
    idx = torch.zeros(1, 1, 8, 1, device="cuda", dtype=torch.int32)
    before = native.launch_count()
    for call in (lambda: native.nsa_compress(r(1, 64, 2, 8), 32, 0), lambda: native.nsa_compress(r(1, 64, 2, 8), 0, 16),
                 lambda: native.nsa_compress(r(1, 64, 2, 8), 32, -16), lambda: native.union_blocks(idx, 0, 1), lambda: native.union_blocks(idx, 256, 1),
                 lambda: native.gated_rms_norm(r(4, 8), r(4, 16)[:, 8:8], r(8))):
        with pytest.raises((ValueError, RuntimeError)):
            call()
    assert native.launch_count() == before


def test_arguments_of_the_wrong_kind_are_refused(native):
    r = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)                # noqa: E731
    f = lambda *s: torch.zeros(*s, device="cuda")                                      # noqa: E731
    hyper = (1, 1e-3, .9, .95, 1e-8, 0.0, None)
    item = (r(256), r(256), f(256), f(256), None, None)
    before = native.launch_count()
    for call, error in ((lambda: native.adamw_multi([], *hyper), IndexError), (lambda: native.adamw8bit_multi([], *hyper, 256), IndexError),
                        (lambda: native.adamw_multi([item[:5]], *hyper), ValueError), (lambda: native.adamw_multi([3], *hyper), TypeError),
                        (lambda: native.adamw_multi([(3,) + item[1:]], *hyper), TypeError), (lambda: native.adamw_multi(3, *hyper), TypeError),
                        (lambda: native._h().multi_linear_fwd(r(256, 64), (r(64, 64), 3)), TypeError)):
        with pytest.raises(error):
            call()
    assert native.launch_count() == before
    ref = torch.ones(256, device="cuda")
    for kind in (list, tuple):                       # any sequence of sequences
        p, g = ref.clone(), ref.clone()
        native.adamw_multi(kind([kind([p, g, f(256), f(256), None, None])]), *hyper)
        assert native.launch_count() > before and (p < 1).all()


def test_flags_of_any_kind(native):
    g = torch.Generator("cuda").manual_seed(0)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16().requires_grad_()   # noqa: E731
    x, w, q, k, a, b = r(1, 20, 64), r(64, 4), r(1, 20, 4, 64), r(1, 20, 2, 64), r(64, 40).detach(), r(64, 24).detach()
    for on in (True, False):
        for op, inputs in ((lambda f: native.causal_conv1d(x, w, None, f), (x, w)), (lambda f: native.attention(q, k, k, f), (q, k))):
            want = [y := op(on), *torch.autograd.grad(y, inputs, torch.ones_like(y))]
            for flag in (np.bool_(on), float(on), int(on), torch.tensor(on)):
                got = [y := op(flag), *torch.autograd.grad(y, inputs, torch.ones_like(y))]
                assert all(torch.equal(s, t) for s, t in zip(got, want))
        out = torch.ones(40, 24, device="cuda")
        want = native.gemm(a, b, True, True, out=out.clone(), accumulate=on)
        assert torch.equal(native.gemm(a, b, np.True_, np.True_, out=out.clone(), accumulate=np.bool_(on)), want)


def test_more_than_64_projections_of_one_input(native):
    g = torch.Generator("cuda").manual_seed(0)
    x = torch.randn(200, 64, device="cuda", generator=g).bfloat16().requires_grad_()
    ws = [torch.randn(8, 64, device="cuda", generator=g).bfloat16().requires_grad_(i > 3) for i in range(67)]
    ys = native.multi_linear(x, ws)
    wanted = [w for w in ws if w.requires_grad]
    got = torch.autograd.grad(ys, wanted, [torch.ones_like(y) for y in ys])
    one = torch.autograd.grad(native.linear(x, wanted[0]), wanted[0], torch.ones_like(ys[0]))[0]
    assert all(torch.equal(w, one) for w in got)         # all of them x summed over its rows
