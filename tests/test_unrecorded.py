"""Which calls of a differentiable op go past autograd (native._run): those that leave nothing to record, and no transform's,
forward-mode derivative's, tracer's or compiler's."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.autograd import forward_ad

from nsa_optim_b200.ops import native


class _Double(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, factor):
        y = factor * x
        ctx.save_for_backward(x)
        ctx.mark_non_differentiable(y)
        return y


@pytest.fixture
def applied(monkeypatch):
    """The calls that reached autograd."""
    calls = []

    def apply(x, factor):
        calls.append(factor)
        return factor * x

    monkeypatch.setattr(_Double, "apply", apply)
    return calls


def test_nothing_to_record(applied):
    x, w = torch.ones(3), torch.ones(3, requires_grad=True)
    for call in (lambda: native._run(_Double, x, 2.0), lambda: torch.no_grad()(lambda: native._run(_Double, w, 2.0))(),
                 lambda: torch.inference_mode()(lambda: native._run(_Double, w, 2.0))()):
        y = call()
        assert torch.equal(y, torch.full((3,), 2.0)) and y.grad_fn is None and not y.requires_grad
    assert applied == []


def test_recorded(applied):
    w = torch.ones(3, requires_grad=True)
    native._run(_Double, w, 2.0)
    native._run(_Double, torch.ones(3) * w, 3.0)
    with torch.no_grad(), torch.enable_grad():
        native._run(_Double, w, 4.0)
    assert applied == [2.0, 3.0, 4.0]


@pytest.mark.parametrize("grad", [True, False])
def test_transforms_see_the_function(applied, monkeypatch, grad):
    # with inputs that no gradient is wanted for: what makes the call go to autograd is the transform alone
    x = torch.ones(2, 3)
    with torch.set_grad_enabled(grad):
        torch.func.vmap(lambda t: native._run(_Double, t, 1.0))(x)
        torch.func.grad(lambda t: native._run(_Double, x, 2.0).sum() * t)(torch.ones(()))
        torch.func.jvp(lambda t: native._run(_Double, t, 3.0), (x,), (x,))
        with forward_ad.dual_level():
            native._run(_Double, forward_ad.make_dual(x, x), 4.0)
        torch.jit.trace(lambda t: native._run(_Double, t, 5.0), (x,), check_trace=False)
        monkeypatch.setattr(torch.compiler, "is_compiling", lambda: True)
        native._run(_Double, x, 6.0)
    assert applied == [1.0, 2.0, 3.0, 4.0, 5.0, 6.0]


@pytest.mark.parametrize("elsewhere", [None, "b", "dt_bias", "A_log"])
def test_gates_of_tensors_on_several_devices_are_left_to_pytorch(monkeypatch, elsewhere):
    calls = []
    monkeypatch.setattr(native, "_h", lambda: type("Host", (), {"gates": lambda self, *a: calls.append(a) or "launched"})())
    with FakeTensorMode():                               # stand-ins for tensors of a GPU
        t = {n: torch.empty(*s, dtype=torch.bfloat16, device="cpu" if n == elsewhere else "cuda:0")
             for n, s in (("a", (1, 4, 8)), ("b", (1, 4, 8)), ("dt_bias", (8,)), ("A_log", (8,)))}
    assert native.delta_gates(**t) == (None if elsewhere else "launched")
    del t["b"]
    assert native.step_sizes(t["a"], t["dt_bias"], t["A_log"]) == (None if elsewhere in ("dt_bias", "A_log") else "launched")
    assert len(calls) == (2 if elsewhere is None else elsewhere == "b")
