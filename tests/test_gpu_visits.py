"""How many query tiles a CTA of the dK / dV kernels takes is read from the environment once a backward, in Python: lists and kernel agree on it, and
the gradients do not depend on it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("visits", ["1", "5", "64"])
def test_read_once_and_honoured(native, monkeypatch, visits):
    T, Hq = 2100, 32
    g = torch.Generator("cuda").manual_seed(0)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16().requires_grad_()      # noqa: E731
    x, gates, dy = [mk(1, T, h, 128) for h in (Hq, 1, 1)], mk(1, T, 3 * Hq), mk(1, T, Hq, 128).detach()
    t = torch.arange(T, device="cuda") // 64
    idx = torch.stack([t, t // 2, torch.zeros_like(t)], -1)[None, None].int()
    calls = {"selected": (lambda: native.selected_attention(*x, idx), x), "range": (lambda: native.attention(*x), x),
             "nsa": (lambda: native.nsa_attention(*x, None, None, None, gate_logits=gates), x + [gates])}
    ys = {n: f() for n, (f, _) in calls.items()}
    want = {n: torch.autograd.grad(y, calls[n][1], dy, retain_graph=True) for n, y in ys.items()}
    read = []

    class Environ(dict):
        def get(self, name, default=None):
            read.append(name)
            return super().get(name, default)

    monkeypatch.setattr(native.os, "environ", Environ({"NSA_B200_KV_VISITS": visits, "NSA_B200_KV_VISITS_SEL": visits}))
    for n, y in ys.items():
        read.clear()
        got = torch.autograd.grad(y, calls[n][1], dy, retain_graph=True)
        assert sorted(r for r in read if "VISITS" in r) == ["NSA_B200_KV_VISITS"] * (n != "selected") + ["NSA_B200_KV_VISITS_SEL"] * (n != "range")
        for a, b in zip(got, want[n]):           # fp32 sums in another order, rounded to bf16: an ulp (2^-8) at a tie, 2^-9 in the mean at most
            assert (a.double() - b.double()).norm() <= 2 ** -9 * b.double().norm()
    native.check_status()
