"""Gated delta rule at the sizes where the chunk kernels can go wrong: shorter than a chunk, around chunk ends, one value
tile, values wider than one launch, unaligned and strided inputs, gates that decay fast or grow, no gradient."""
import pytest
import torch

from nsa_optim_b200.ops import oracle, torch_impl

pytestmark = pytest.mark.gpu


def _inputs(B, T, H, V, decay, dtype=torch.float32):
    torch.manual_seed(T + V)
    q, k = (oracle.l2_norm(torch.randn(B, T, H, 128, device="cuda")).bfloat16() for _ in range(2))
    v = torch.randn(B, T, H, V, device="cuda").bfloat16()
    g = (-torch.rand(B, T, H, device="cuda") * decay).to(dtype)
    beta = torch.rand(B, T, H, device="cuda").to(dtype)
    return [q, k, v, g, beta]


def _check(native, inputs, tol=2e-2):
    leaves = [t.detach().requires_grad_() for t in inputs]
    o = native.gated_delta_rule(*leaves)
    do = torch.randn_like(o)
    got = [o.detach()] + list(torch.autograd.grad(o, leaves, do))
    ref = [t.detach().double().requires_grad_() for t in inputs]
    # the chunked PyTorch form in the inputs' widest precision
    r = torch_impl.gated_delta_rule(*[t.float() for t in ref], chunk=64)
    want = [r.detach()] + list(torch.autograd.grad(r, ref, do.float()))
    for name, a, b in zip(("o", "dq", "dk", "dv", "dg", "dbeta"), got, want):
        assert a.shape == b.shape
        # operands are rounded to bf16 (2^-9 each) a handful of times on the way to any output
        err = (a.double() - b.double()).norm() / (b.double().norm() + 1e-12)
        assert err < tol, (name, float(err))
    return got[0]


@pytest.mark.parametrize("B,T,H,V", [(1, 1, 1, 64), (2, 63, 3, 128), (1, 64, 2, 256), (2, 65, 1, 256), (1, 130, 5, 192), (1, 300, 2, 640)])
def test_gdn_sizes(native, B, T, H, V):
    _check(native, _inputs(B, T, H, V, 0.3))


@pytest.mark.parametrize("T,H,V", [(1300, 16, 64), (1283, 15, 320), (1000, 20, 512)])
def test_gdn_more_chunks_than_sms(native, T, H, V):
    # two chunks' gradients share an SM; one, five and eight slices of the values
    _check(native, _inputs(1, T, H, V, 0.3))


@pytest.mark.parametrize("decay", [0.0, 8.0, -0.01])       # no decay, e^-500 across a chunk, slow growth
def test_gdn_gates(native, decay):
    _check(native, _inputs(1, 200, 2, 256, decay))


def test_gdn_strided_unaligned_bf16_gates(native):
    q, k, v, g, beta = _inputs(1, 100, 2, 128, 0.3, torch.bfloat16)
    flat = torch.zeros(q.numel() + 4, device="cuda", dtype=torch.bfloat16)
    q2 = flat[4:].view(q.shape).copy_(q)                                          # 8-byte aligned only
    v2 = v.transpose(1, 2).contiguous().transpose(1, 2)
    a = _check(native, [q2, k, v2, g, beta])
    with torch.no_grad():
        b = native.gated_delta_rule(q, k, v, g, beta)
    assert torch.equal(a, b)


def test_gdn_more_chunks_than_a_second_grid_dimension_holds(native):
    # 65540 chunks of 64 tokens.  Decays of e^-3 per chunk at least: what is more than a hundred chunks away is gone, so both ends
    # equal runs over the ends alone.
    T, n, keep = 65540 * 64, 128 * 64, 16 * 64
    inputs = _inputs(1, T, 1, 64, 0.2)
    inputs[3] -= 0.05

    def run(ts, dy):
        leaves = [t.detach().requires_grad_() for t in ts]
        o = native.gated_delta_rule(*leaves)
        return [o.detach()] + list(torch.autograd.grad(o, leaves, dy))

    dy = torch.randn(1, T, 1, 64, device="cuda").bfloat16()
    whole = run(inputs, dy)
    for part, kept in ((slice(0, n), slice(0, keep)), (slice(T - n, T), slice(n - keep, n))):
        ends = run([t[:, part] for t in inputs], dy[:, part])
        for a, b in zip(whole, ends):
            a, b = a[:, part][:, kept].double(), b[:, kept].double()
            assert b.norm() > 0 and (a - b).norm() <= 2 ** -8 * b.norm()
