"""Step sizes and gates in one launch: the bits of PyTorch's functions for all kinds of values, layouts and parameter types, and which calls
take it."""
import pytest
import torch

from nsa_optim_b200 import ops
from nsa_optim_b200.ops import torch_impl

pytestmark = pytest.mark.gpu


def _inputs(B, T, H, dtype):
    g = torch.Generator("cuda").manual_seed(T + H)
    wide = (torch.randn(B, T, 2 * H + 24, device="cuda", generator=g) * 12).bfloat16()
    flat = wide.view(-1)
    odd = torch.tensor([0.0, -0.0, 20.0, 20.125, -20.0, 88.5, -104.0, float("inf"), float("-inf"), float("nan")], device="cuda").bfloat16()
    flat[::7][:10] = odd[:flat[::7][:10].numel()]
    bias, A_log = ((torch.randn(H, device="cuda", generator=g) * s).to(dtype) for s in (2, 3))
    return wide[..., 8:8 + H], wide[..., 16 + H:16 + 2 * H], bias, A_log


@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 3, 5), (1, 1000, 64), (2, 77, 8), (1, 20000, 48)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dense", [True, False])
def test_same_bits(native, B, T, H, dtype, dense):
    a, b, bias, A_log = _inputs(B, T, H, dtype)
    if dense:
        a, b = a.contiguous(), b.transpose(0, 1).contiguous().transpose(0, 1)          # b: another order of its rows
    before = native.launch_count()
    got = ops.step_sizes(a, bias, A_log) + ops.delta_gates(a, b, bias, A_log)
    assert native.launch_count() == before + 2
    for x, y in zip(got, torch_impl.step_sizes(a, bias, A_log) + torch_impl.delta_gates(a, b, bias, A_log)):
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x.nan_to_num(123.0), y.nan_to_num(123.0))


def test_recorded_calls_stay_differentiable(native):
    a, b, bias, A_log = (t.detach().requires_grad_() for t in _inputs(1, 40, 6, torch.float32))
    before = native.launch_count()
    for out, args in ((ops.step_sizes(a, bias, A_log), (a, bias, A_log)), (ops.delta_gates(a, b, bias, A_log), (a, b, bias, A_log))):
        assert all(g is not None for g in torch.autograd.grad([t.nan_to_num().sum() for t in out], args))
    assert native.launch_count() == before
    with torch.no_grad():
        ops.step_sizes(a, bias, A_log)
    assert native.launch_count() == before + 1


def test_parameters_on_the_host_are_treated_as_by_pytorch(native):
    a, b, bias, A_log = _inputs(1, 40, 6, torch.float32)
    before = native.launch_count()
    for call in (lambda: ops.step_sizes(a, bias.cpu(), A_log), lambda: ops.delta_gates(a, b, bias.cpu(), A_log),
                 lambda: ops.delta_gates(a, b, bias, A_log.cpu())):
        with pytest.raises(RuntimeError):
            call()
    assert all(x.device == y.device and torch.equal(x.nan_to_num(123.0), y.nan_to_num(123.0))
               for x, y in zip(ops.step_sizes(a, bias, A_log.cpu()), torch_impl.step_sizes(a, bias, A_log.cpu())))
    assert native.launch_count() == before
