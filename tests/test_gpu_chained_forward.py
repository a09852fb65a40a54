"""Small forwards launch their kernels chained (a kernel may start before the one ahead of it has
ended).  Nothing may be seen early: inputs written on the stream just before the call, outputs read
just after it, the same through a captured graph, and forwards on two streams at once.  The output of
each case is also compared with the oracle, since every run here takes the chained path."""

import pytest
import torch

from moe_bench_b200 import problem as P
from moe_bench_b200.plugin import get_implementation
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# precision, tokens, experts, hidden, intermediate: 16-bit; fp8 with tokens on the columns; fp8 128-row
# tiles; sorts of one block (up to 1024 assignments) and of several, last size of chaining (8192).  fp8
# with tokens on the columns and a sort of several blocks has every kernel chained to the one ahead of it:
# count, scatter, quantise, row gather, gate/up, down, combine.
CASES = [("bf16", 1, 64, 1024, 512), ("fp16", 512, 16, 1024, 512), ("bf16", 513, 16, 1024, 512),
         ("bf16", 1025, 8, 1024, 512), ("fp8", 3, 64, 1024, 512), ("fp8", 200, 4, 1024, 512),
         ("fp8", 1024, 32, 1024, 512), ("bf16", 128, 32, 512, 256), ("bf16", 129, 32, 512, 256),
         ("fp8", 129, 256, 512, 256), ("fp8", 600, 256, 256, 128), ("fp8", 600, 512, 512, 256),
         ("fp8", 1024, 640, 256, 128)]


def _setup(precision, tokens, experts, seed, hidden=1024, intermediate=512):
    cfg = P.MoEBenchConfig(hidden_size=hidden, intermediate_size=intermediate, num_experts=experts, topk=min(8, experts),
                           world_size=1, precision=P.Precision(precision), seed=seed, device=DEV)
    prob = P.make_problem(cfg, tokens)
    impl = get_implementation("b200")
    impl.setup(prob)
    return impl, prob


def _variants(prob, n=4):
    gen = torch.Generator(device=DEV).manual_seed(9)
    xs = [torch.randn(prob.hidden_states.shape, device=DEV, generator=gen).to(prob.hidden_states.dtype) for _ in range(n)]
    ids = [prob.topk_ids.roll(i + 1, 0) for i in range(n)]
    return xs, ids


@pytest.mark.parametrize("precision,tokens,experts,hidden,intermediate", CASES)
def test_inputs_written_on_the_stream(precision, tokens, experts, hidden, intermediate):
    impl, prob = _setup(precision, tokens, experts, 1, hidden, intermediate)
    first = impl.run(prob)
    res = O.verify_output(precision, first, O.reference_moe(prob))
    # three roundings to 8 (11) significand bits, 2^-9 (2^-12) each, relative to a sum of k terms; fp8 keeps
    # bf16 activations and both sides quantise the same values
    assert res.passed and res.rel_err < (1.5e-3 if precision == "fp16" else 1e-2), (res.message, res.rel_err)
    xs, ids = _variants(prob)
    want = []
    for x, i in zip(xs, ids):
        prob.hidden_states.copy_(x)
        prob.topk_ids.copy_(i)
        torch.cuda.synchronize()
        want.append(impl.run(prob).clone())
        torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for x, i in zip(xs, ids):
            prob.hidden_states.copy_(x)
            prob.topk_ids.copy_(i)
            got.append(impl.run(prob).clone())
        for g, w in zip(got, want):
            assert torch.equal(g, w)
    assert impl.device_status() == 0

    graph = torch.cuda.CUDAGraph()
    outs = [torch.empty_like(w) for w in want]
    with torch.cuda.graph(graph):
        for x, i, o in zip(xs, ids, outs):
            prob.hidden_states.copy_(x)
            prob.topk_ids.copy_(i)
            o.copy_(impl.run(prob))
    for _ in range(3):
        for o in outs:
            o.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert torch.equal(o, w)
    del graph


def test_two_streams():
    jobs = [_setup("bf16", 5, 32, 2), _setup("fp8", 150, 4, 3)]
    want = [impl.run(prob).clone() for impl, prob in jobs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(20):
        for k, (impl, prob) in enumerate(jobs):
            with torch.cuda.stream(streams[k]):
                got[k].append(impl.run(prob).clone())
    torch.cuda.synchronize()
    for k in range(2):
        assert jobs[k][0].device_status() == 0
        assert all(torch.equal(g, want[k]) for g in got[k])
