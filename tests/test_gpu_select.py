"""Top-n selection against a plain sort: numbers of blocks around a warp's 32, ties, zeros of either sign, infinities and NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _plain(imp, sel_block, top_n):
    B, H, T, nS = imp.shape
    out = torch.full((B, H, T, top_n), -1, dtype=torch.int32)
    rows = imp.tolist()
    for b in range(B):
        for h in range(H):
            for t in range(T):
                own = min(t // sel_block, nS - 1)
                forced = list(dict.fromkeys(j for j in (0, own, own - 1) if j >= 0))[:top_n]
                r = rows[b][h][t]
                free = [j for j in range(1, own - 1) if not math.isnan(r[j]) and r[j] != -math.inf]
                free.sort(key=lambda j: -r[j])             # stable: the lower index first
                got = forced + free[: top_n - len(forced)]
                out[b, h, t, : len(got)] = torch.tensor(got, dtype=torch.int32)
    return out


@pytest.mark.parametrize("nS,top_n", [(1, 4), (3, 2), (31, 16), (33, 16), (64, 1), (100, 16), (257, 40)])
def test_select_against_a_sort(native, nS, top_n):
    torch.manual_seed(nS)
    T, sel_block = 4 * nS + 3, 4
    imp = torch.randint(-3, 9, (1, 2, T, nS)).float() / 4  # many ties
    imp[torch.rand_like(imp) < 0.1] = -0.0
    for value in (math.inf, -math.inf, math.nan):
        imp[torch.rand_like(imp) < 0.03] = value
    got = native.nsa_select(imp.cuda(), sel_block, top_n).cpu()
    assert torch.equal(got.int(), _plain(imp, sel_block, top_n))
