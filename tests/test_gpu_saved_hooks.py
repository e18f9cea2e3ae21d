"""Saved-tensor hooks: with activations kept on the host the saved tensors come back dense, whatever their strides were."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases(native):
    torch.manual_seed(0)
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()                       # noqa: E731
    B, T, H = 2, 200, 3
    wide = rnd(B, T, H * 64 + 256 + 64)                                              # one projection, sliced
    dt, A = torch.rand(B, T, H, device="cuda") * 0.1, -torch.rand(H, device="cuda") - 1
    yield ("ssd", lambda x, dt, A, b, c, d: native.ssd_scan(x, dt, A, b, c, d),
           [wide[..., :H * 64].unflatten(-1, (H, 64)), dt, A, wide[..., H * 64:H * 64 + 128].unsqueeze(2),
            wide[..., H * 64 + 128:H * 64 + 256].unsqueeze(2), torch.ones(H, device="cuda")])
    gate = rnd(300, 1024 + 64)[:, 64:]
    for before in (True, False):
        yield ("gated norm", lambda x, g, w, before=before: native.gated_rms_norm(x, g, w, 1e-5, before),
               [rnd(300, 1024), gate, rnd(1024)])
    yield "conv1d", lambda x, w, b: native.causal_conv1d(x, w, b), [rnd(B, T, 264)[..., 8:136], rnd(128, 4), rnd(128)]
    gu = rnd(300, 2 * 512)
    yield "swiglu", lambda g, u: native.swiglu(g, u), [gu[:, :512], gu[:, 512:]]
    yield "linear", lambda x, w: native.linear(x, w), [rnd(256, 192)[:, 64:], rnd(64, 128)]
    yield ("gdn", lambda q, k, v, g, b: native.gated_delta_rule(q, k, v, g, b),
           [torch.nn.functional.normalize(rnd(1, T, H, 128).float(), dim=-1).bfloat16() for _ in range(2)]
           + [rnd(1, T, H, 128), -torch.rand(1, T, H, device="cuda"), torch.rand(1, T, H, device="cuda")])
    qkv = rnd(1, T, 8 + 2, 128)
    yield ("nsa", lambda q, k, v, g: native.nsa_attention(q, k, v, None, None, None, gate_logits=g),
           [*qkv.split([8, 1, 1], 2), rnd(1, T, 24)])


def test_saved_tensors_kept_on_the_host(native):
    for name, op, inputs in _cases(native):
        leaves = [t.detach().requires_grad_() for t in inputs]
        y = op(*leaves)
        dy = torch.randn_like(y)
        want = torch.autograd.grad(y, leaves, dy)
        with torch.autograd.graph.save_on_cpu():
            got = torch.autograd.grad(op(*leaves), leaves, dy)
        for a, b in zip(got, want):
            assert a.shape == b.shape and torch.equal(a, b), name
