"""The layer workloads whose speed is tracked: what a program that serves or benchmarks an
MoE layer has this package do, through the calls it would make itself.

A *layer* case is one forward through the compute-only plugin (``get_implementation("b200")``:
``setup`` once, ``run`` per step), an *ep_scheme* case one forward through the distributed
plugin at world size 1 (staging, barriers, dispatch, expert GEMMs and combine of one rank), a
*router* case the gating front end alone (``capi.route_topk``: softmax, top-k, renormalise).

Inputs come from the package's own seeded generator (N(0,1) tokens, N(0,1)/sqrt(fan-in)
weights, routing drawn by distribution), so they have the values and the load shapes that the
benchmark and the tests use.  The model shapes:

  dsv32      hidden 7168, intermediate 2048, 256 experts, top-8, all experts on this GPU
  dsv32_ep8  one rank of 8 of the same layer, expert parallel: 32 local experts, the tokens of
             all ranks, an expert map that sends 7/8 of the assignments elsewhere
  dsv32_tp8  one rank of 8, tensor parallel: every expert with an intermediate slice of 256
  default    the benchmark's default configuration: hidden 4096, intermediate 3072 over 8
             tensor-parallel ranks (384 each), 64 experts, top-8
  default_1  the same without the split (intermediate 3072 on this GPU)
"""

import math

import torch

from moe_bench_b200 import capi
from moe_bench_b200.plugin import get_implementation
from moe_bench_b200.problem import MoEBenchConfig, ParallelMode, Precision, RoutingConfig, Distribution, make_problem
from moe_bench_b200.scheme import DistContext, get_scheme

DEVICE = "cuda:0"

# name -> (hidden, intermediate, experts, topk, parallel mode, ranks the layer is split over)
SHAPES = {
    "dsv32": (7168, 2048, 256, 8, "tp", 1),
    "dsv32_ep8": (7168, 2048, 256, 8, "ep", 8),
    "dsv32_tp8": (7168, 2048, 256, 8, "tp", 8),
    "dsv32_32e": (7168, 2048, 32, 8, "ep", 1),  # the 32 experts of one of 8 ranks, run as a world of one
    "default": (4096, 3072, 64, 8, "tp", 8),
    "default_1": (4096, 3072, 64, 8, "tp", 1),
}
# tokens a case of each shape may have
TOKENS = {
    "dsv32": (1, 8192),
    "dsv32_ep8": (8, 32768),
    "dsv32_tp8": (8, 16384),
    "dsv32_32e": (1, 4096),
    "default": (1, 4096),
    "default_1": (1, 4096),
}
ROUTER_TOKENS = (1, 16384)
ROUTER_EXPERTS = (32, 64, 256)


def _layer(name, shape, precision, tokens, routing="uniform", entry="layer"):
    case = {"entry": entry, "shape": shape, "precision": precision, "tokens": tokens, "routing": routing}
    return dict(case, name=name) if name else case


def _router(name, tokens, experts, topk=8):
    case = {"entry": "router", "tokens": tokens, "experts": experts, "topk": topk}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one sequence being decoded: eight experts' weights are streamed once, launches count
        _layer("decode_1_bf16", "dsv32", "bf16", 1),
        # a small decode batch in the deployed precision
        _layer("decode_8_fp8", "dsv32", "fp8", 8),
        # a full decode batch: every expert is touched by a handful of rows, HBM-bound
        _layer("decode_128_bf16", "dsv32", "bf16", 128),
        # the same in fp8, with an odd number of sequences in flight
        _layer("decode_131_fp8", "dsv32", "fp8", 131),
        # a prefill chunk: 64 rows per expert, between weight streaming and arithmetic
        _layer("prefill_2048_fp8", "dsv32", "fp8", 2048),
        # a large prefill, the benchmark's headline workload, in both precisions
        _layer("prefill_8192_bf16", "dsv32", "bf16", 8192),
        _layer("prefill_8192_fp8", "dsv32", "fp8", 8192),
        # expert-parallel serving, 4096 tokens on each of 8 ranks: this rank's 32 experts with
        # about 1024 rows each, 7/8 of the assignments belong to other ranks
        _layer("ep8_rank_32768_fp8", "dsv32_ep8", "fp8", 32768),
        # tensor-parallel serving: thin slices of every expert, a reduction dimension of 256
        _layer("tp8_rank_4096_bf16", "dsv32_tp8", "bf16", 4096),
        # the distributed plugin's own path, 1024 tokens for 32 experts
        _layer("ep_scheme_1024_fp8", "dsv32_32e", "fp8", 1024, entry="ep_scheme"),
        # the default configuration with a ragged batch, a skewed load and fp16 tensors
        _layer("default_777_fp16_skewed", "default", "fp16", 777, routing="skewed"),
        # the gating front end of a large prefill
        _router("router_8192", 8192, 256),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer"] * 8 + ["ep_scheme", "router"])
    if kind == "router":
        return _router(None, _log_uniform(rng, *ROUTER_TOKENS), rng.choice(ROUTER_EXPERTS))
    shape = "dsv32_32e" if kind == "ep_scheme" else rng.choice(
        ["dsv32", "dsv32", "dsv32", "dsv32_ep8", "dsv32_tp8", "default", "default_1"])
    precision = rng.choice(["bf16", "bf16", "fp8", "fp8", "fp16"])
    routing = rng.choice(["uniform", "uniform", "uniform", "balanced", "skewed"])
    return _layer(None, shape, precision, _log_uniform(rng, *TOKENS[shape]), routing, kind)


def _config(case, seed):
    hidden, inter, experts, topk, mode, world = SHAPES[case["shape"]]
    return MoEBenchConfig(
        hidden_size=hidden, intermediate_size=inter, num_experts=experts, topk=topk,
        parallel_mode=ParallelMode(mode), world_size=world, precision=Precision(case["precision"]),
        routing=RoutingConfig(distribution=Distribution(case["routing"])), seed=seed, device=DEVICE)


def prepare(case, seed):
    """The problem bundle and the plugin set up for it (workspace and output buffer), or the logits."""
    if case["entry"] == "router":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)
        logits = torch.randn(case["tokens"], case["experts"], device=DEVICE, dtype=torch.float32, generator=gen)
        return {"logits": logits, "topk": case["topk"]}
    problem = make_problem(_config(case, seed), case["tokens"])
    if case["entry"] == "ep_scheme":
        scheme = get_scheme("b200")
        scheme.setup(problem, DistContext(rank=0, world_size=1, local_rank=0, device=torch.device(DEVICE)))
        return {"scheme": scheme}
    impl = get_implementation("b200")
    impl.setup(problem)
    return {"impl": impl, "problem": problem}


def run(state):
    if "logits" in state:
        return capi.route_topk(state["logits"], state["topk"])
    if "scheme" in state:
        return state["scheme"].run()
    return state["impl"].run(state["problem"])


def _touched_experts(case, experts, local, topk):
    """Expected number of this rank's experts that get a row (rank 0 owns the first ``local``)."""
    tokens, routing = case["tokens"], case["routing"]
    if routing == "balanced":
        return min(local, tokens * topk)
    p = [(e + 1.0) ** -1.0 if routing == "skewed" else 1.0 for e in range(experts)]
    total = sum(p)
    return sum(1.0 - (1.0 - min(1.0, topk * v / total)) ** tokens for v in p[:local])


def work(case):
    if case["entry"] == "router":
        t, e, k = case["tokens"], case["experts"], case["topk"]
        return {"bytes": 4 * t * e + 8 * t * k, "flops": 4 * t * e}
    hidden, inter, experts, topk, mode, world = SHAPES[case["shape"]]
    local = experts // world if mode == "ep" else experts
    n = inter // world if mode == "tp" else inter
    tokens = case["tokens"]
    share = 1.0
    if mode == "ep" and world > 1:
        share = 1.0 / world
        if case["routing"] == "skewed":  # the first experts are the popular ones; at most one row per token each
            p = [1.0 / (e + 1) for e in range(experts)]
            share = sum(min(1.0 / topk, v / sum(p)) for v in p[:local])
    rows = tokens * topk * share
    weight_bytes = 1 if case["precision"] == "fp8" else 2
    touched = _touched_experts(case, experts, local, topk)
    return {
        "bytes": int(touched * 3 * n * hidden * weight_bytes + 2 * tokens * hidden * 2 + 8 * tokens * topk),
        "flops": int(6 * n * hidden * rows),
    }


def _dequant_weight(w, scale):
    """One expert's weight in 64 bits; fp8: every 128x128 block times its scale."""
    if scale is None:
        return w.double()
    blocks = scale.double().repeat_interleave(128, 0)[: w.shape[0]].repeat_interleave(128, 1)[:, : w.shape[1]]
    return w.to(torch.float32).double() * blocks


def _quantised(x):
    """Activations as the fp8 path defines them: e4m3 with one scale per row and 128 columns,
    a power of two where the reference's quantiser makes it one."""
    groups = x.reshape(x.shape[0], -1, 128)
    scale = groups.abs().amax(-1, keepdim=True).clamp(min=1e-10) / 448.0
    if capi.reference_fp8_scale_format() == "ue8m0":
        scale = torch.exp2(torch.ceil(torch.log2(scale)))
    q = (groups / scale).clamp(-448.0, 448.0).float().to(torch.float8_e4m3fn)
    return (q.float().double() * scale).reshape(x.shape)


def exact(case, seed):
    """What ``run`` returns, in 64 bits: the router's ids and weights, or the layer's output,
    expert by expert (fp8: on the quantised activations that the precision means)."""
    if case["entry"] == "router":
        logits = prepare(case, seed)["logits"].double()
        best, ids = torch.sort(logits, dim=1, descending=True, stable=True)
        best, ids = best[:, : case["topk"]], ids[:, : case["topk"]]
        return ids.to(torch.int32), torch.softmax(best, 1)
    problem = make_problem(_config(case, seed), case["tokens"])
    fp8 = case["precision"] == "fp8"
    x = problem.hidden_states.double()
    if fp8:
        x = _quantised(x)
    ids = problem.topk_ids.long()
    if problem.expert_map is not None:
        ids = problem.expert_map.long()[ids]
    out = torch.zeros_like(x)
    n = problem.w1.shape[1] // 2
    for e in range(problem.w1.shape[0]):
        token, slot = torch.nonzero(ids == e, as_tuple=True)
        if token.numel() == 0:
            continue
        w1 = _dequant_weight(problem.w1[e], problem.quant_config.w1_scale[e] if fp8 else None)
        w2 = _dequant_weight(problem.w2[e], problem.quant_config.w2_scale[e] if fp8 else None)
        h = x[token] @ w1.t()
        act = torch.nn.functional.silu(h[:, :n]) * h[:, n:]
        if fp8:
            act = _quantised(act.bfloat16().double())  # bf16 activations are part of the precision
        out.index_add_(0, token, problem.topk_weights[token, slot].double()[:, None] * (act @ w2.t()))
    return out


def tolerance(case):
    if case["entry"] == "router":
        # fp32 softmax over a few selected logits; the ids are exact
        return {"rel": 1e-6, "max": 2e-6, "differ": 0.0}
    # Intermediate activations, weighted rows and the output are rounded to the 16-bit type (fp8
    # keeps bf16 activations).  Against the same layer in 64 bits: fp16 rel 3.6e-4, max 1.8e-3;
    # bf16 and fp8 rel 2.9e-3, max 2.7e-2 (of the rms).  About four times that.
    if case["precision"] == "fp16":
        return {"rel": 1.5e-3, "max": 8e-3}
    return {"rel": 1.2e-2, "max": 1.1e-1}
