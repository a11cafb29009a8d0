"""The work this library is measured on: what a serving process has it do, on one GPU.

Four kinds of pass, all through public entry points:

* ``comm``: dispatch -> synthetic expert -> combine on a :class:`Context` (the headline benchmark's
  step): eager with a retained workspace, as tickets without one, or replayed from a CUDA graph;
* ``ranks``: the same for a group of several ranks, every rank's share inside single launches
  (:class:`EmulatedGroup`) - the multi-rank kernels, protocol and all, on one GPU;
* ``layer``: the full MoE layer (dispatch -> grouped SwiGLU experts -> combine);
* ``experts``: the expert runner alone on the padded batch one rank of a larger group receives.

Shapes: hidden 7168 with top-8 and 2048-wide experts (the DeepSeek-V3-shaped benchmark; 32 experts are
one rank's share of 256) and hidden 2048 with 128 experts (the Qwen3-30B-A3B-shaped one). Decode
batches run from graphs, prefill batches eagerly. A program keeps its context, workspace, weights
and expert runner; inputs are new for every seed.
"""

from __future__ import annotations

import atexit
import math
import random
import weakref
from collections import OrderedDict

import torch
import torch.distributed as dist

from ep_xpress_b200 import Config, Context, EmulatedGroup, get_nccl_comm_handle
from ep_xpress_b200.models import SwiGLUMoELayer
from ep_xpress_b200.ops import GroupedSwiGLU, scale_rows

_V3 = dict(hidden=7168, topk=8)
_QWEN = dict(hidden=2048, topk=8, experts=128)


def _case(kind, name=None, *, tokens, hidden, topk, experts, inter=0, world=1, mode="eager", routing="uniform",
          pad=0.0, ids="int64", rounding="auto", pair=True):
    case = dict(kind=kind, tokens=tokens, hidden=hidden, topk=topk, experts=experts, inter=inter, world=world,
                mode=mode, routing=routing, pad=pad, ids=ids, rounding=rounding, pair=pair)
    return case if name is None else dict(name=name, **case)


def listed():
    return [
        # The smallest call there is: one token, eager. Launches and host time count.
        _case("comm", "comm-v3-1", tokens=1, experts=256, **_V3),
        # The decode benchmark: 128 tokens, the layer replayed as one CUDA graph.
        _case("comm", "comm-v3-128-graph", tokens=128, experts=256, mode="graph", **_V3),
        # The headline prefill step.
        _case("comm", "comm-v3-4096", tokens=4096, experts=256, **_V3),
        # Tickets without a workspace, int32 ids, skewed routing, padded tokens (id -1), one rounding.
        _case("comm", "comm-qwen3-3001-async", tokens=3001, mode="async", routing="zipf", pad=0.1, ids="int32",
              rounding="single", **_QWEN),
        # A decode step of a four-rank group (count exchange, peer rows, mailbox combine).
        _case("ranks", "ranks4-v3-128-graph", tokens=128, experts=256, world=4, mode="graph", **_V3),
        # Decode of an eight-rank group on skewed routes, an odd batch with padded tokens.
        _case("ranks", "ranks8-qwen3-67-graph", tokens=67, world=8, mode="graph", routing="zipf", pad=0.1, **_QWEN),
        # A prefill chunk of a four-rank group.
        _case("ranks", "ranks4-v3-1024", tokens=1024, experts=256, world=4, **_V3),
        # The full layer for one token (a lone request): eight experts' weights.
        _case("layer", "layer-v3-1", tokens=1, experts=32, inter=2048, **_V3),
        # The full layer at the decode batch: every expert's weights, few rows each.
        _case("layer", "layer-v3-128-graph", tokens=128, experts=32, inter=2048, mode="graph", **_V3),
        # The full layer at the prefill batch: bound by the tensor cores.
        _case("layer", "layer-v3-4096", tokens=4096, experts=32, inter=2048, **_V3),
        # Many small experts, skewed and odd: ragged tiles.
        _case("layer", "layer-qwen3-1021", tokens=1021, inter=768, routing="zipf", pad=0.1, **_QWEN),
        # The runner with its default options on the batch one of eight ranks receives: a padded
        # capacity, most slots belonging to other ranks.
        _case("experts", "experts-ep8-509", tokens=509, hidden=2048, topk=8, experts=16, inter=768, world=8, pair=False),
    ]


def _spread(rng, low, high):
    """Log-uniform whole number, odd ones as likely as even ones."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.5))))))


def draw(rng: random.Random):
    kind = rng.choice(["comm", "comm", "ranks", "ranks", "layer", "layer", "experts"])
    common = dict(topk=rng.choice([1, 2, 4, 6, 8, 8, 8]), routing=rng.choice(["uniform", "zipf"]),
                  pad=round(rng.choice([0.0, rng.uniform(0.0, 0.3)]), 3), ids=rng.choice(["int64", "int32"]),
                  rounding=rng.choice(["auto", "auto", "single"]))
    if kind == "comm":
        tokens = _spread(rng, 1, 8192)
        return _case(kind, tokens=tokens, hidden=8 * rng.randint(128, 896), experts=rng.choice([64, 128, 256]),
                     mode=rng.choice(["graph", "eager", "async"] if tokens <= 256 else ["eager", "async"]), **common)
    if kind == "ranks":
        world = rng.choice([2, 4, 8])
        tokens = _spread(rng, 1, 4096 // world)
        return _case(kind, tokens=tokens, hidden=8 * rng.randint(128, 896), experts=rng.choice([64, 128, 256]),
                     world=world, mode="graph" if tokens <= 256 and rng.random() < 0.7 else "eager", **common)
    hidden, inter = 256 * rng.randint(4, 28), 128 * rng.randint(2, 16)
    experts = _spread(rng, 8, 64 if inter <= 1024 else 32)
    tokens = _spread(rng, 1, 4096)
    if kind == "layer":
        return _case(kind, tokens=tokens, hidden=hidden, experts=experts, inter=inter,
                     mode="graph" if tokens <= 256 and rng.random() < 0.7 else "eager", pair=rng.random() < 0.8, **common)
    world = rng.choice([2, 4, 8])
    return _case(kind, tokens=tokens, hidden=hidden, experts=experts, inter=inter, world=world,
                 pair=rng.random() < 0.5, **common)


# ---- what a serving program keeps ------------------------------------------------------------------
def _comm():
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1,
                                device_id=torch.device("cuda", 0))
        atexit.register(_leave)
    return get_nccl_comm_handle(dist.group.WORLD)


def _leave():
    _programs.clear()
    dist.destroy_process_group()


class _Program:
    """Context (or group), workspace and weights of one configuration."""

    def __init__(self, case):
        tokens, hidden, topk, inter = case["tokens"], case["hidden"], case["topk"], case["inter"]
        world, experts = case["world"], case["experts"]
        cfg = Config(hidden_size=hidden, topk=topk, max_tokens_per_rank=tokens, timeout_seconds=10.0,
                     gpu_pool_budget_bytes=64 << 30, combine_rounding=case["rounding"])
        if inter:
            g = torch.Generator(device="cuda").manual_seed(1234)
            w13 = torch.empty((experts, 2 * inter, hidden), dtype=torch.bfloat16, device="cuda").normal_(0, 0.02, generator=g)
            w2 = torch.empty((experts, hidden, inter), dtype=torch.bfloat16, device="cuda").normal_(0, 0.02, generator=g)
        if case["kind"] == "experts":
            # A rank's fair share of the group's (token, slot) pairs with room for skew.
            rows = world * tokens
            self.experts = GroupedSwiGLU(w13, w2, max_rows=rows, topk=topk, pair_ctas=case["pair"],
                                         max_local_pairs=min(rows * topk, 6 * tokens * topk + 1024))
        elif case["kind"] == "ranks":
            self.group = EmulatedGroup(world, [e * world // experts for e in range(experts)], cfg)
            self.slot = self.group.create_slot()
            weakref.finalize(self, self.group.close).atexit = False
        else:
            self.context = Context(_comm(), [0] * experts, cfg)
            weakref.finalize(self, self.context.close).atexit = False
            if case["mode"] == "graph":
                self.context.enable_cuda_graph()
            if case["kind"] == "layer":
                self.layer = SwiGLUMoELayer(self.context, w13, w2, pair_ctas=case["pair"])
            elif case["mode"] != "async":
                self.workspace = self.context.create_workspace(tokens, tokens)


_programs = OrderedDict()


def _program(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _programs:
        while len(_programs) >= 2:
            _programs.popitem(last=False)
        _programs[key] = _Program(case)
    _programs.move_to_end(key)
    return _programs[key]


# ---- inputs -------------------------------------------------------------------------------------
def _popularity(routing, experts, permutation):
    p = [1.0 / (i + 1) ** 1.2 for i in range(experts)] if routing == "zipf" else [1.0] * experts
    total = sum(p)
    return [p[permutation[e]] / total for e in range(experts)]


def _routes(case, experts, rank, seed, g):
    """Expert ids without replacement per token and normalised sigmoid weights; the last
    ``pad`` share of the tokens is padding (every id -1)."""
    tokens, topk = case["tokens"], case["topk"]
    permutation = list(range(experts))
    random.Random(seed).shuffle(permutation)
    p = torch.tensor(_popularity(case["routing"], experts, permutation), device="cuda")
    uniform = torch.rand((tokens, experts), generator=g, device="cuda").clamp_(1e-7, 1 - 1e-7)
    ids = (p.log() - (-uniform.log()).log()).topk(topk, dim=1).indices        # Gumbel: sampling without replacement
    weights = torch.sigmoid(torch.randn((tokens, topk), generator=g, device="cuda"))
    weights = weights / weights.sum(dim=1, keepdim=True)
    ids[_live(case):] = -1
    return ids, weights


def _live(case):
    return max(1, case["tokens"] - int(case["tokens"] * case["pad"]))


def _payload(case, g):
    return torch.empty((case["tokens"], case["hidden"]), dtype=torch.bfloat16, device="cuda").normal_(generator=g)


class _State:
    pass


def _received(case, seed):
    """The batch rank 0 of ``world`` ranks receives: rows in (source, token) order, then padding."""
    world, experts = case["world"], case["experts"]
    rows, ids, weights = [], [], []
    for rank in range(world):
        g = torch.Generator(device="cuda").manual_seed(seed * 1009 + rank)
        i, w = _routes(case, world * experts, rank, seed, g)
        x = _payload(case, g)
        i = torch.where(i < experts, i, -1)
        here = (i >= 0).any(dim=1)
        rows.append(x[here]), ids.append(i[here]), weights.append(w[here])
    capacity, valid = world * case["tokens"], sum(len(r) for r in rows)
    hidden = torch.zeros((capacity, case["hidden"]), dtype=torch.bfloat16, device="cuda")
    local = torch.full((capacity, case["topk"]), -1, dtype=torch.int64, device="cuda")
    scale = torch.zeros((capacity, case["topk"]), dtype=torch.float32, device="cuda")
    hidden[:valid], local[:valid], scale[:valid] = torch.cat(rows), torch.cat(ids), torch.cat(weights)
    return hidden, local, scale, torch.tensor([valid], dtype=torch.int32, device="cuda")


def prepare(case, seed):
    s = _State()
    s.kind, s.mode, s.program = case["kind"], case["mode"], _program(case)
    s.inputs, s.graph = [], None
    if s.kind == "experts":
        s.inputs = _received(case, seed)
        s.out = torch.zeros_like(s.inputs[0])
        return s
    for rank in range(case["world"]):
        g = torch.Generator(device="cuda").manual_seed(seed * 1009 + rank)
        ids, weights = _routes(case, case["experts"], rank, seed, g)
        s.inputs.append((_payload(case, g), ids.to(getattr(torch, case["ids"])), weights))
    s.outs = [torch.empty_like(x) for x, _, _ in s.inputs] if s.kind == "ranks" else None
    if s.mode == "graph":
        _capture(s)
    return s


def _capture(s):
    """The decode path: warm once, then capture the whole pass on a side stream."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _pass(s)
    side.synchronize()
    if s.kind != "ranks":
        s.program.context.prepare_graph_capture()
    s.graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s.graph, stream=side):
        s.outputs = _pass(s)
    torch.cuda.current_stream().wait_stream(side)


# ---- one pass ------------------------------------------------------------------------------------
def run(state):
    if state.graph is None:
        return _pass(state)
    if state.kind != "ranks":
        state.program.context.prepare_graph_replay()
    state.graph.replay()
    return state.outputs


def _pass(s):
    if s.kind == "experts":
        hidden, ids, weights, count = s.inputs
        return s.program.experts(hidden, ids, weights, count, out=s.out)
    if s.kind == "ranks":
        group, slot = s.program.group, s.program.slot
        xs, ids, weights = zip(*s.inputs)
        batches = group.dispatch(slot, xs, ids, weights)
        partials = [group.scale_rows(batch) for batch in batches]
        outs = group.combine(slot, partials, [len(x) for x in xs], outs=s.outs)
        return [(b.hidden, b.local_ids, b.weights, b.inverse, b.valid_count) for b in batches], outs
    x, ids, weights = s.inputs[0]
    if s.kind == "layer":
        return s.program.layer(x, ids, weights)
    ep = s.program.context
    if s.mode == "async":
        batch = ep.dispatch_async(x, ids, weights, tag="layer").wait()
        out = ep.combine_async(scale_rows(ep, batch), batch.handle, tag="layer").wait()
    else:
        batch = ep.dispatch_on_stream(x, ids, weights, workspace=s.program.workspace)
        out = ep.combine_on_stream(scale_rows(ep, batch), batch.handle)
    return batch.hidden, batch.local_ids, batch.weights, batch.handle.inverse_map, batch.valid_count, out


# ---- what a pass cannot do without ----------------------------------------------------------------
def _expected(case, experts, group_size, tokens):
    """(Mean destinations per token, mean number of one destination's experts that get a token) for
    experts in ``group_size``-sized blocks: inclusion odds of sampling without replacement."""
    topk = min(case["topk"], experts)
    permutation = list(range(experts))
    random.Random(0).shuffle(permutation)
    p = _popularity(case["routing"], experts, permutation)
    low, high = 0.0, 1e9
    for _ in range(200):
        rate = (low + high) / 2
        low, high = (rate, high) if sum(-math.expm1(-rate * q) for q in p) < topk else (low, rate)
    blocks = [p[i:i + group_size] for i in range(0, experts, group_size)]
    destinations = sum(-math.expm1(-rate * sum(block)) for block in blocks)
    used = sum(-math.expm1(-rate * tokens * q) for q in p) / len(blocks)
    return destinations, used


def work(case):
    """Inputs read once and outputs written once, call by call: dispatch reads the activations and
    routes and writes the received rows with their routes; the expert reads and writes those rows;
    combine reads them and writes the tokens. Experts read the weights of the experts in use."""
    tokens, hidden, topk, world = case["tokens"], case["hidden"], case["topk"], case["world"]
    live, row = _live(case), hidden * 2
    id_bytes = 4 if case["ids"] == "int32" else 8
    expert_bytes = 3 * hidden * case["inter"] * 2
    if case["kind"] == "experts":
        destinations, used = _expected(case, world * case["experts"], case["experts"], world * live)
        rows, pairs = destinations * live, live * topk        # one rank's mean share of world * live tokens
        return {"bytes": rows * (2 * row + topk * 12) + used * expert_bytes, "flops": pairs * 6 * hidden * case["inter"]}
    destinations, used = _expected(case, case["experts"], case["experts"] // world, live)
    rows = world * live * min(destinations, world)
    received = row + topk * 12 + 16                           # activations, ids, weights, inverse entry
    dispatch = world * tokens * topk * (id_bytes + 4) + world * live * row + rows * received
    combine = rows * row + world * tokens * row
    if case["kind"] == "layer":
        return {"bytes": dispatch + rows * (2 * row + topk * 12) + used * expert_bytes + combine,
                "flops": live * topk * 6 * hidden * case["inter"]}
    return {"bytes": dispatch + rows * (2 * row + topk * 12) + combine, "flops": 0.0}


def tolerance(case):
    """Communication moves bytes and adds in a fixed order and rounding: exact. The experts round
    activations and every slot's result to BF16 and may sum their products in another order: against
    the same layer in FP64 the listed and drawn cases show rel 2.5e-3 to 2.9e-3 and max 0.010 to
    0.027; about four times that."""
    if case["kind"] in ("comm", "ranks"):
        return "exact"
    return {"rel": 1e-2, "max": 0.1}
