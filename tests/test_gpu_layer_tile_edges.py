"""16-bit layer where its kernels change shape: short K in the down GEMM with one accumulator pair
(segments past 128 rows; fewer K steps than pipeline stages), ragged feature blocks, single and many
experts, and all forms of the combine (few tokens / enough to fill the GPU, wide / narrow rows), all
rows local or one rank's share of them."""

import pytest
import torch

from moe_bench_b200 import problem as P
from moe_bench_b200.plugin import get_implementation
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [
    # tokens, hidden, intermediate, experts, topk, distribution, mode, ranks
    (150, 320, 64, 1, 1, "uniform", "tp", 1),      # one expert, 150 rows, one K step
    (300, 576, 128, 4, 2, "uniform", "tp", 1),     # two K steps, ragged last 256-feature block
    (1100, 512, 192, 8, 3, "skewed", "tp", 1),     # segments of 50 to 1000 rows, three K steps
    (700, 768, 256, 5, 2, "single", "tp", 1),      # four K steps, more than the ring holds; empty experts
    (2400, 320, 64, 8, 5, "uniform", "ep", 4),     # narrow groups, a quarter of the rows local
    (2367, 64, 64, 40, 9, "balanced", "tp", 1),    # too few tokens for narrow groups, k > 8, 8 vectors per row
    (40, 2048, 512, 640, 8, "uniform", "tp", 1),   # tile lookup over more experts than 32 x 16
    (2368, 64, 64, 40, 9, "balanced", "tp", 1),    # combine in groups of 8 lanes, one vector each; k > 8
    (2367, 192, 64, 16, 3, "uniform", "ep", 2),    # the last size of whole warps for rows that do not fill them
    (2371, 576, 64, 8, 5, "uniform", "ep", 4),     # two vectors a lane, ragged last run, absent rows
    (1187, 1152, 64, 24, 17, "uniform", "tp", 1),  # the same over two sweeps of 128, k > 16
    (2368, 896, 64, 8, 2, "uniform", "tp", 1),     # whole warps, the last quarter of the lanes' vectors half empty
]


@pytest.mark.parametrize("precision", ["bf16", "fp16"])
@pytest.mark.parametrize("tokens,hidden,inter,experts,topk,dist,mode,world", CASES)
def test_layer_matches_oracle(precision, tokens, hidden, inter, experts, topk, dist, mode, world):
    cfg = P.MoEBenchConfig(hidden_size=hidden, intermediate_size=inter, num_experts=experts, topk=topk,
                           parallel_mode=P.ParallelMode(mode), world_size=world, precision=P.Precision(precision),
                           routing=P.RoutingConfig(distribution=P.Distribution(dist)), seed=tokens, device=DEV)
    prob = P.make_problem(cfg, tokens)
    impl = get_implementation("b200")
    impl.setup(prob)
    out = impl.run(prob)
    assert impl.device_status() == 0
    res = O.verify_output(precision, out, O.reference_moe(prob))
    # three roundings to 8 (11) significand bits, 2^-9 (2^-12) each, relative to a sum of k terms
    assert res.passed and res.rel_err < (1e-2 if precision == "bf16" else 1.5e-3), (res.message, res.rel_err)
    assert torch.equal(out, impl.run(prob))
