"""route_topk at the edges of its register variants (1, 2, 4, 8, 16, 32 logits per lane) and on
rows with masked, NaN, infinite and tied logits: the ids are the oracle's, and so always topk
different experts of the row, also where fewer than topk logits are usable."""

import math

import pytest
import torch

from moe_bench_b200 import capi
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _select(row, k):
    """Largest logit first, lowest index on ties, -0 == +0, NaN after -inf (the oracle's stable sort);
    weights: softmax over the selected, where a NaN weighs nothing."""
    ids = O.route_topk(row[None], k)[0][0].tolist()
    picked = torch.nan_to_num(row[ids], nan=-math.inf, posinf=math.inf, neginf=-math.inf)
    p = torch.exp(picked - picked[0])
    return ids, p / p.sum()


@pytest.mark.parametrize("experts,topk", [(1, 1), (31, 8), (32, 32), (33, 8), (64, 8), (65, 8), (128, 8), (129, 33),
                                          (256, 8), (257, 8), (512, 9), (513, 64), (1024, 8)])
def test_route_topk_register_variants(experts, topk):
    gen = torch.Generator().manual_seed(experts * 31 + topk)
    logits = torch.randn(15, experts, generator=gen)
    logits[1] = 0.0
    logits[2] = (logits[2] * 2).round() / 2        # many ties
    logits[3, ::2] = -0.0
    logits[3, 1::2] = 0.0                          # -0 and +0 tie: lowest index
    logits[4, experts // 2 :] = -math.inf          # masked experts
    logits[5, : experts - 1] = math.nan
    logits[6, -1] = 3.0e38
    logits[7] = -3.0e38
    logits[9] = math.nan                           # nothing usable: ids 0 .. topk-1
    logits[10] = -math.inf
    logits[11, ::3] = -math.inf                    # -inf before NaN, both by index
    logits[11, 1::3] = math.nan
    logits[12] = -math.inf
    logits[12, -1] = 5.0                           # one usable logit, the last
    logits[13] = math.nan
    logits[13, experts // 3] = -math.inf
    logits[14, 0] = math.inf
    ids, w = capi.route_topk(logits.to(DEV), topk)
    for t in range(15):
        o_ids, o_w = _select(logits[t], topk)
        assert len(set(o_ids)) == topk and 0 <= min(o_ids) and max(o_ids) < experts
        assert ids[t].tolist() == o_ids, t
        # exp and the sum of up to 64 terms in fp32: (64 + 4) * 2^-24 relative
        torch.testing.assert_close(w[t].cpu(), o_w, atol=1e-6, rtol=5e-6, equal_nan=True)
