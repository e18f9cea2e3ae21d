"""Mamba-2 scan forward and backward where the chunk, state and head-sum kernels can go wrong: shorter than a chunk, around chunk
ends, head counts off the eight heads of a summation block and odd, two sequences, no skip weight, strided inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(x, dt, A, Bm, Cm, D):
    """The recurrence in 64 bits, one step at a time."""
    h = x.new_zeros(x.shape[0], x.shape[2], x.shape[3], Bm.shape[-1])
    ys = []
    for t in range(x.shape[1]):
        h = h * torch.exp(dt[:, t] * A)[..., None, None] + (dt[:, t, :, None] * x[:, t])[..., None] * Bm[:, t, 0][:, None, None, :]
        ys.append(torch.einsum("bhpn,bn->bhp", h, Cm[:, t, 0]))
    y = torch.stack(ys, 1)
    return y if D is None else y + x * D[:, None]


@pytest.mark.parametrize("B,T,H,skip", [(1, 1, 1, True), (2, 100, 3, False), (1, 128, 8, True), (2, 129, 9, True), (1, 300, 24, False)])
def test_ssd_sizes(native, B, T, H, skip):
    torch.manual_seed(T)
    xbc = torch.nn.functional.silu(torch.randn(B, T, H * 64 + 256, device="cuda")).bfloat16()
    dt = torch.nn.functional.softplus(torch.randn(B, T, H, device="cuda") - 3)
    leaves = [xbc[..., :H * 64].view(B, T, H, 64), dt, -torch.rand(H, device="cuda") * 15 - 1, xbc[..., H * 64:H * 64 + 128].view(B, T, 1, 128),
              xbc[..., H * 64 + 128:].view(B, T, 1, 128)] + ([torch.rand(H, device="cuda") + 0.5] if skip else [])
    leaves = [t.detach().requires_grad_() for t in leaves]
    dy = (torch.randn(B, T, H, 64, device="cuda") + 0.5).bfloat16()
    y = native.ssd_scan(*leaves)
    got = [y.detach()] + list(torch.autograd.grad(y, leaves, dy))
    ref = [t.detach().double().requires_grad_() for t in leaves]
    r = _reference(*ref, *([] if skip else [None]))
    want = [r.detach()] + list(torch.autograd.grad(r, ref, dy.double()))
    for name, a, b in zip(("y", "dx", "ddt", "dA", "dB", "dC", "dD"), got, want):
        assert a.shape == b.shape
        # bf16 operands and per-head terms: 2^-9 each, a few of them, averaged over the sums
        assert (a.double() - b).norm() < 1e-2 * b.norm() + 1e-6, name


# 32 sequences x heads and more: the states come from one walk over the chunks (one chunk, as many as it has stages, more); runs of
# (chunk, head) items that end inside a chunk, at its end, and go over several
@pytest.mark.parametrize("B,T,H,skip", [(32, 5, 1, True), (1, 256, 32, True), (2, 384, 16, False), (1, 513, 48, True), (2, 700, 70, True),
                                        (1, 1100, 33, False), (1, 1100, 70, False)])
def test_ssd_walk_and_runs(native, B, T, H, skip):
    test_ssd_sizes(native, B, T, H, skip)


@pytest.mark.parametrize("B,T,H,one", [(1, 300, 1, True), (1, 1000, 1, False), (1, 1000, 48, False), (1, 777, 64, True), (1, 16384, 48, False),
                                       (1, 16384, 64, True)])
def test_choice_of_state_kernels(native, B, T, H, one):
    assert bool(native.load().nsa_ssd_states_in_one(B, T, H)) == one              # times of both: see there


# A step that forgets everything, or is not finite, at each place of the four that a lane scans, in the second chunk: what comes
# before it does not see it.  One head (a kernel per chunk) and many (one walk over the chunks).
@pytest.mark.parametrize("at", [168, 169, 171])
@pytest.mark.parametrize("T,H", [(300, 40), (1500, 1)])
def test_steps_before_a_long_one(native, T, H, at):
    torch.manual_seed(at)
    x, Bm, Cm, dy = (torch.randn(1, T, h, n, device="cuda").bfloat16() for h, n in ((H, 64), (1, 128), (1, 128), (H, 64)))
    dt, A = torch.rand(1, T, H, device="cuda") * 0.1 + 0.01, -torch.ones(H, device="cuda")
    plain = native.ssd_scan(x, dt, A, Bm, Cm)
    for bad in (float("inf"), float("nan"), 1e6):
        dt[:, at] = bad
        assert torch.equal(native.ssd_scan(x, dt, A, Bm, Cm)[:, :at], plain[:, :at]), bad
    leaves = [t.detach().requires_grad_() for t in (x, dt, A, Bm, Cm)]
    got = torch.autograd.grad(native.ssd_scan(*leaves), leaves, dy)
    ref = [t.detach().double().requires_grad_() for t in leaves]
    want = torch.autograd.grad(_reference(*ref, None), ref, dy.double())
    for name, i in (("dx", 0), ("dB", 3), ("dC", 4)):
        a, b = got[i][:, :at].double(), want[i][:, :at]
        assert (a - b).norm() < 1e-2 * b.norm(), name                                # as above


# dA holds the sums over the tokens from each one on of dy.y - x.dx, times its step.  Terms of different kernels cancel in them: up to the
# rounding of the bf16 operands, averaged over a row's products, where the kernels agree on the decays.  With a step of 1e6 the sums
# of steps are multiples of 1/16 and decays rounded in different ways are up to 6 % apart.  One walk over the chunks, and two kernels.
@pytest.mark.parametrize("T,H,at", [(700, 64, 168), (700, 64, 171), (2000, 64, 300), (1500, 2, 171)])
def test_decays_agree_behind_a_long_step(native, T, H, at):
    torch.manual_seed(at)
    x, Bm, Cm, dy = (torch.randn(1, T, h, n, device="cuda").bfloat16() for h, n in ((H, 64), (1, 128), (1, 128), (H, 64)))
    dt, A = torch.rand(1, T, H, device="cuda") * 0.1 + 0.01, -torch.ones(H, device="cuda")
    dt[:, at] = 1e6
    leaves = [t.detach().requires_grad_() for t in (x, dt, A, Bm, Cm)]
    dA = torch.autograd.grad(native.ssd_scan(*leaves), leaves, dy)[2]
    ref = [t.detach().double().requires_grad_() for t in leaves]
    y = _reference(*ref, None)
    want = torch.autograd.grad(y, ref, dy.double())[2]
    terms = (y.detach() * dy.double()).sum(-1)[0, at:]                              # (tokens, H): what cancels
    assert ((dA - want).abs() <= 1e6 * 2 ** -9 * 128 ** -0.5 * terms.norm(dim=0)).all()


@pytest.mark.parametrize("nc,E", [(1, 7), (7, 12), (8, 64), (9, 1000), (30, 8192)])
@pytest.mark.parametrize("back", [False, True])
def test_state_pass(native, nc, E, back):
    from ctypes import c_int, c_long, c_void_p
    torch.manual_seed(nc)
    B, H = 2, 3
    S, gamma = torch.randn(B, nc, H, E, device="cuda"), torch.rand(B, nc, H, device="cuda")
    out, out_bf = torch.empty_like(S), torch.empty(S.shape, device="cuda", dtype=torch.bfloat16)
    p = lambda t: c_void_p(t.data_ptr())                                            # noqa: E731
    dims = (c_int(B), c_int(nc), c_int(H), c_long(E), native._stream())
    if back:
        native._check(native.load().nsa_ssd_state_bwd(p(S), p(gamma), p(out), p(out_bf), *dims))
    else:
        native._check(native.load().nsa_ssd_state_fwd(p(S), p(gamma), p(out), p(out_bf), c_void_p(0), *dims))
    st, want = torch.zeros(B, H, E, device="cuda", dtype=torch.float64), torch.empty(S.shape, device="cuda", dtype=torch.float64)
    for c in (reversed(range(nc)) if back else range(nc)):
        want[:, c] = st
        st = gamma[:, c, :, None].double() * st + S[:, c].double()
    assert (out.double() - want).abs().max() <= 1e-5 * want.abs().max() + 1e-12     # one fp32 rounding per chunk, decaying
    assert torch.equal(out_bf, out.to(torch.bfloat16))


def test_ssd_more_chunks_than_a_second_grid_dimension_holds(native):
    # 65540 chunks of 128 tokens, one head.  Decays of e^-6 per chunk at least: what is more than fifty chunks away is gone, so
    # both ends equal runs over the ends alone.
    torch.manual_seed(0)
    T, n, keep = 65540 * 128 - 28, 100 * 128, 16 * 128
    xbc = torch.randn(1, T, 320, device="cuda", dtype=torch.bfloat16)
    dy = torch.randn(1, T, 1, 64, device="cuda", dtype=torch.bfloat16)
    dt, A, D = torch.rand(1, T, 1, device="cuda") * 0.05 + 0.05, -torch.ones(1, device="cuda"), torch.ones(1, device="cuda")

    def run(part):
        x = xbc[:, part]
        leaves = [t.detach().requires_grad_() for t in (x[..., :64].unflatten(-1, (1, 64)), dt[:, part], A,
                                                        x[..., 64:192].unsqueeze(2), x[..., 192:].unsqueeze(2), D)]
        y = native.ssd_scan(*leaves)
        dx, ddt, _, dB, dC, dD = torch.autograd.grad(y, leaves, dy[:, part])
        return [y.detach(), dx, dB, dC, ddt], dD

    whole, dD = run(slice(0, T))
    want = (xbc[..., :64].double() * dy[:, :, 0].double()).sum()
    assert abs(float(dD - want)) <= 1e-3 * T ** 0.5 * 8                              # a sum of 64 T products of size one
    tail = T - n + 28                                                                # on a chunk boundary
    for part, kept, outputs in ((slice(0, n), slice(0, keep), 4), (slice(tail, T), slice(n - keep - 128, None), 5)):
        # ddt is a sum over all later tokens, whose rounding is not that of a shorter run's: compared at the end only
        for a, b in list(zip(whole, run(part)[0]))[:outputs]:
            a, b = a[:, part][:, kept].double(), b[:, kept].double()
            assert b.shape[1] >= 1 and b.norm() > 0 and (a - b).norm() <= 2 ** -8 * b.norm()


def test_state_pass_of_few_elements_is_a_short_chain(native):
    # 1000 chunks of 3 x 63 elements: what one step takes. 32 us; 87 with addresses computed per access
    from ctypes import c_int, c_long, c_void_p
    p = lambda t: c_void_p(t.data_ptr())                                            # noqa: E731
    B, nc, H, E = 1, 1000, 3, 63
    S, gamma = torch.randn(B, nc, H, E, device="cuda"), torch.rand(B, nc, H, device="cuda")
    out = torch.empty(S.shape, device="cuda", dtype=torch.bfloat16)
    times = []
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            native._check(native.load().nsa_ssd_state_fwd(p(S), p(gamma), c_void_p(0), p(out), c_void_p(0), c_int(B), c_int(nc), c_int(H),
                                                          c_long(E), native._stream()))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) / 20 * 1e3)
    assert min(times[2:]) <= 60, times


# Partial sums per token on both sides of the rule for how many are in flight: room for 1, 2, 4, 5, 13, 17 and 40
@pytest.mark.parametrize("B,T,H", [(1, 130, 1), (16, 900, 8), (7, 1000, 24), (1, 140, 5), (1, 1500, 24), (2, 129, 17), (1, 128, 40)])
def test_ssd_partial_sums(native, B, T, H):
    test_ssd_sizes(native, B, T, H, True)


def test_no_items(native):
    # sizes that nothing can be launched for are refused by the kernels' entry points; asking what they need is no crash
    for sizes in ((0, 100, 8), (1, 0, 8), (1, 100, 0)):
        assert native.load().nsa_ssd_grad_slots(*sizes) >= 0
        assert native.load().nsa_ssd_states_in_one(*sizes) in (0, 1)
