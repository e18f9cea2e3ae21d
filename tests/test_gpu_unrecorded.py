"""Every op without gradients, where it goes past autograd, against the same op recorded: the same bits, and no graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases(native):
    g = torch.Generator("cuda").manual_seed(0)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()                  # noqa: E731
    f = lambda *s: torch.rand(*s, device="cuda", generator=g)                              # noqa: E731
    ids = torch.randint(0, 64, (2, 9), device="cuda", generator=g)
    cos, sin = f(70, 64), f(70, 64)
    q, k, v, gl = r(1, 200, 16, 128), r(1, 200, 2, 128), r(1, 200, 2, 128), r(1, 200, 48)
    idx = torch.zeros(1, 2, 200, 1, dtype=torch.int32, device="cuda")
    return {
        "linear": (native.linear, r(40, 256), r(128, 256)),
        "multi_linear": (lambda x, a, b: native.multi_linear(x, (a, b)), r(40, 256), r(128, 256), r(64, 256)),
        "rms_norm": (native.rms_norm, r(33, 256), r(256)),
        "rms_norm_skip": (native.rms_norm_skip, r(33, 256), r(256)),
        "add_rms_norm": (native.add_rms_norm, r(33, 256), r(33, 256), r(256)),
        "gated_rms_norm": (native.gated_rms_norm, r(33, 256), r(33, 256), r(256)),
        "l2_norm": (native.l2_norm, r(33, 128)),
        "swiglu": (native.swiglu, r(33, 256), r(33, 256)),
        "rope": (lambda x: native.rope(x, cos, sin), r(2, 70, 4, 128)),
        "causal_conv1d": (native.causal_conv1d, r(2, 50, 64), r(64, 4), r(64)),
        "embedding": (lambda w: native.embedding(ids, w), r(64, 128)),
        "linear_cross_entropy": (lambda h, w: native.linear_cross_entropy(h, w, ids.reshape(-1)), r(18, 128), r(64, 128)),
        "attention": (native.attention, q, k, v),
        "selected_attention": (lambda *x: native.selected_attention(*x, idx), q, k, v),
        "nsa_compress": (lambda x: native.nsa_compress(x, 32, 16), k),
        "nsa_attention": (lambda a, b, c, d: native.nsa_attention(a, b, c, None, None, None, gate_logits=d), q, k, v, gl),
        "gated_delta_rule": (native.gated_delta_rule, r(1, 100, 2, 128) / 12, r(1, 100, 2, 128) / 12, r(1, 100, 2, 128), -f(1, 100, 2), f(1, 100, 2)),
        "ssd_scan": (native.ssd_scan, r(1, 200, 3, 64), f(1, 200, 3), -f(3) - 0.1, r(1, 200, 1, 128), r(1, 200, 1, 128), f(3)),
    }


def test_same_bits(native):
    for name, (op, *inputs) in _cases(native).items():
        leaves = [t.clone().requires_grad_() for t in inputs]
        recorded = op(*leaves)
        with torch.no_grad():
            off = op(*leaves)
        none = op(*inputs)
        for a, b, c in zip(*(t if isinstance(t, tuple) else (t,) for t in (recorded, off, none))):
            assert a.grad_fn is not None and b.grad_fn is None and c.grad_fn is None and not c.requires_grad, name
            assert torch.equal(a.detach(), b) and torch.equal(b, c), name
