"""Native sparse attention as one autograd node, and block selection at the edges of its register sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native():
    from nsa_optim_b200 import ops
    return ops.native_module()


@pytest.mark.parametrize("nS", [1, 128, 129, 256, 257, 512, 513, 1024, 1025])
def test_selection_at_the_edges_of_the_register_sizes(native, nS):
    T = nS * 4 - 1
    imp = torch.rand(1, 1, T, nS, device="cuda", generator=torch.Generator("cuda").manual_seed(nS))
    imp[:, :, ::7] = imp[:, :, ::7].mul(4).round()          # ties: the lower index wins
    imp[:, :, ::11] = 0
    got = native.nsa_select(imp, 4, 16)
    own = (torch.arange(T, device="cuda") // 4)[:, None]
    j = torch.arange(nS, device="cuda")[None]
    score = imp.masked_fill((j == 0) | (j == own) | (j == own - 1), float("inf")).masked_fill(j > own, float("-inf"))
    top = score.sort(dim=-1, descending=True, stable=True)
    want = top.indices[..., :16].masked_fill(top.values[..., :16] == float("-inf"), -1).to(torch.int32)
    want = torch.nn.functional.pad(want, (0, 16 - want.shape[-1]), value=-1)
    assert torch.equal(got.sort(-1).values, want.sort(-1).values)


def _separate(native, q, k, v, gates, window):
    """The branches as nodes of their own: the sums and additions happen outside the kernels."""
    kc, vc = native.nsa_compress(k, 32, 16), native.nsa_compress(v, 32, 16)
    sc, nS = q.shape[-1] ** -0.5, -(-q.shape[1] // 64)
    o1, L1 = native._Attn.apply(q, kc, vc, True, 0, sc, 16, 31, None)
    with torch.no_grad():
        tiles = native._nsa_select_tiles(q, kc, L1, nS, 16, 32, 64, 16, sc)
    o2 = native._Attn.apply(q, k, v, True, 0, sc, 1, 0, tiles)[0]
    o3 = native._Attn.apply(q, k, v, True, window, sc, 1, 0, None)[0]
    return native._GateCombineLogits.apply(o1, o2, o3, gates)


# 32 tokens: no second compressed key; group 32 with window 700: several CTAs of the window branch meet in one key block
@pytest.mark.parametrize("B,T,Hq,Hkv,window,extra", [(1, 32, 8, 1, 512, 0), (2, 333, 16, 2, 64, 0), (1, 1000, 32, 2, 512, 40),
                                                     (1, 2100, 32, 1, 700, 0), (1, 700, 32, 4, 700, 0)])
def test_one_node_matches_separate_branches(native, B, T, Hq, Hkv, window, extra):
    g = torch.Generator("cuda").manual_seed(T)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()     # noqa: E731
    # q, k, v as column groups of one projection: not contiguous
    qkv = mk(B, T, Hq + 2 * Hkv, 128)
    x = [t.detach().requires_grad_() for t in (*qkv.split([Hq, Hkv, Hkv], 2), mk(B, T, 3 * Hq + extra))]
    dy = mk(B, T, Hq, 128)
    y = native.nsa_attention(*x[:3], None, None, None, window=window, gate_logits=x[3])
    got = torch.autograd.grad(y, x, dy, retain_graph=True)
    again = torch.autograd.grad(y, x, dy)
    ref = _separate(native, *x, window)
    want = torch.autograd.grad(ref, x, dy)
    native.check_status()
    assert torch.equal(y, ref) and torch.equal(got[3], want[3])
    for a, b, c in zip(got, want, again):
        # three roundings to bf16 of partial sums (2^-9 each) against one
        assert (a.float() - b.float()).norm() <= 3 * 2 ** -9 * b.float().norm()
        # every token selects block 0, 64 groups of R tokens to a CTA: up to two CTAs add in either order to the same bits
        if T <= 2 * 64 * (128 * Hkv // Hq):
            assert torch.equal(a, c)


@pytest.mark.parametrize("D", [64, 128])
def test_combine_backward_with_and_without_row_sums(native, D):
    g = torch.Generator("cuda").manual_seed(D)
    o1, o2, o3, do = (torch.randn(3, 37, 5, D, device="cuda", generator=g).bfloat16() for _ in range(4))
    gl = torch.randn(3, 37, 15, device="cuda", generator=g).bfloat16()
    plain = native._gate_logits_backward(o1, o2, o3, gl, do)
    sums = [torch.empty(3, 37, 5, device="cuda") for _ in range(3)]
    for a, b in zip(plain, native._gate_logits_backward(o1, o2, o3, gl, do, sums)):
        assert torch.equal(a, b)
    for d, o, s in zip(plain, (o1, o2, o3), sums):
        want = (d.double() * o.double()).sum(-1)
        assert (s.double() - want).abs().max() <= 1e-5 * (d.double() * o.double()).abs().sum(-1).max()    # fp32 sums


def test_combine_backward_without_row_sums_does_not_pay_for_them(native):
    # 2097152 rows of 128: 570 us, 617 with the sums
    o = [torch.randn(65536, 32, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    gl = torch.randn(65536, 96, device="cuda", dtype=torch.bfloat16)
    sums = [torch.empty(65536, 32, device="cuda") for _ in range(3)]

    def fastest(*extra):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(8):
                native._gate_logits_backward(*o[:3], gl, o[3], *extra)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    without, together = fastest(), fastest(sums)
    assert without <= 0.96 * together, (without, together)
