"""Native sparse attention: block selection at the edges of its register sizes."""
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
