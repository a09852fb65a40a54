"""route_topk at the edges of its register variants (1, 2, 4, 8, 16, 32 logits per lane) and on
rows with masked, NaN, infinite and tied logits."""

import math

import pytest
import torch

from moe_bench_b200 import capi

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _select(row, k):
    """The kernel's rule, one row: largest logit first, lowest index on ties, -0 == +0, a NaN is
    never selected, a winner goes on as -inf (so that masked rows run out onto the lowest index)."""
    v = [x for x in row.tolist()]
    ids, picked = [], []
    for _ in range(k):
        best, best_e = -math.inf, 0x7FFFFFFF
        for e, x in enumerate(v):
            if x > best or (x == best and e < best_e):
                best, best_e = x, e
        ids.append(best_e)
        picked.append(best)
        if best_e < len(v):
            v[best_e] = -math.inf
    p = torch.exp(torch.tensor(picked, dtype=torch.float32) - picked[0])
    return ids, p / p.sum()


@pytest.mark.parametrize("experts,topk", [(1, 1), (31, 8), (32, 32), (33, 8), (64, 8), (65, 8), (128, 8), (129, 33),
                                          (256, 8), (257, 8), (512, 9), (513, 64), (1024, 8)])
def test_route_topk_register_variants(experts, topk):
    gen = torch.Generator().manual_seed(experts * 31 + topk)
    logits = torch.randn(9, experts, generator=gen)
    logits[1] = 0.0
    logits[2] = (logits[2] * 2).round() / 2        # many ties
    logits[3, ::2] = -0.0
    logits[3, 1::2] = 0.0                          # -0 and +0 tie: lowest index
    logits[4, experts // 2 :] = -math.inf          # masked experts
    logits[5, : experts - 1] = math.nan
    logits[6, -1] = 3.0e38
    logits[7] = -3.0e38
    ids, w = capi.route_topk(logits.to(DEV), topk)
    for t in range(9):
        o_ids, o_w = _select(logits[t], topk)
        assert ids[t].tolist() == o_ids, t
        # exp and the sum of up to 64 terms in fp32: (64 + 4) * 2^-24 relative
        torch.testing.assert_close(w[t].cpu(), o_w, atol=1e-6, rtol=5e-6, equal_nan=True)
