"""Mamba-2 scan where two CTAs walk the chunks of a head, each with half of the state's rows: two chunks and more than the walk has stages, odd
heads, two sequences, and the last head count that all fit with."""
import pytest
import torch
from test_gpu_ssd_sizes import test_ssd_sizes as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,skip", [(1, 129, 1, True), (1, 256, 5, False), (2, 385, 9, True), (1, 700, 64, True), (2, 770, 37, False),
                                        (1, 897, 48, True), (1, 1000, 74, True), (2, 1665, 32, True)])
def test_halves(native, B, T, H, skip):
    assert native.load().nsa_ssd_states_form(B, T, H) == 2
    _check(native, B, T, H, skip)


# one chunk; more CTAs than SMs; few heads and many chunks, where two kernels are faster
@pytest.mark.parametrize("B,T,H,form", [(1, 128, 64, 1), (1, 1000, 75, 1), (2, 4000, 64, 1), (1, 16384, 24, 0), (1, 16384, 64, 2), (0, 1, 1, 0)])
def test_form(native, B, T, H, form):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert native.load().nsa_ssd_states_form(B, T, H) == form


# the kernels that run: by the time of both forms where heads are few, one walk beyond half as many heads as SMs, a head more than SMs among them
@pytest.mark.parametrize("B,T,H,form", [(1, 300, 1, 2), (1, 1000, 1, 2), (1, 1300, 1, 0), (1, 1000, 48, 2), (1, 777, 64, 2), (1, 4000, 32, 0), (1, 16384, 48, 2),
                                        (1, 300, 75, 1), (1, 16384, 148, 1), (1, 129, 149, 1), (1, 300, 149, 1), (2, 200, 80, 1), (3, 129, 99, 1),
                                        (4, 8000, 80, 1)])
def test_form_by_heads(native, B, T, H, form):
    test_form(native, B, T, H, form)


@pytest.mark.parametrize("B,T,H,skip", [(1, 300, 149, True), (3, 129, 99, False)])
def test_more_heads_than_sms(native, B, T, H, skip):
    _check(native, B, T, H, skip)
