"""The work that users of the sparse decode reader have it do, as cases that can be timed.

Two kinds of case:

* "decode": one decode step through a few MoE layers, each called once through
  `ProgressiveReader.__call__` on its own hidden rows and router outputs.  The layers have
  weights of their own and share one `ReaderWorkspace`, as the layers of a model do; there
  are enough of them that a step's weights come from HBM and not from L2.  `graph` cases
  replay a CUDA graph of the step, which is how a serving engine runs decode; the others
  call the readers eagerly, which is what the vLLM binding of this repository does.
* "sketch": the ternary sketch of a layer's gate/up rows, built on the device
  (`build_sketch_on_device`), which every layer of a model needs once when it is loaded.

Weights, inputs and routing follow the synthetic layers of the benchmark (Gaussian weights;
Gaussian hidden states, with outlier channels, or Student-t; softmax top-k routing, with a
per-expert bias where the load is skewed), drawn on the device from the seed.
"""

from __future__ import annotations

import math

import torch

import cfm_b200  # noqa: F401  (registers the package alias)
from cfm_b200.reader.budget import compile_budget
from cfm_b200.reader.progressive import ProgressiveReader, ReaderWorkspace
from cfm_b200.reader.sketch import block_hadamard_signs, build_sketch_on_device

_DECODE = {
    "kind": "decode", "tokens": 1, "layers": 1, "hidden": 2048, "width": 768, "experts": 128,
    "top_k": 8, "rank": 64, "retention": 0.123046875, "screen_keep": 0.625, "score": "point",
    "activation": "silu", "inputs": "normal", "skewed": False, "renormalize": True,
    "threshold": False, "padding": 0, "ids64": False, "weights16": False,
    "prepare_input": False, "graph": False,
}
_OLMOE = {"width": 1024, "experts": 64, "renormalize": False}
_QWEN3 = {"inputs": "outliers"}
_QWEN35 = {"width": 512, "experts": 256, "inputs": "student_t", "skewed": True}
_WIDE = {"hidden": 4096, "width": 1536, "rank": 128}


def _decode(name: str, *changes: dict, **more: object) -> dict:
    case = {"name": name, **_DECODE}
    for change in (*changes, more):
        case.update(change)
    return case


def listed() -> list[dict]:
    return [
        # One user's chat, called eagerly: a single token through a few OLMoE-shaped layers.
        _decode("olmoe one token eager", _OLMOE, tokens=1, layers=6),
        # The same under a serving engine's captured decode step.
        _decode("qwen3 one token graph", _QWEN3, tokens=1, layers=6, graph=True),
        # A handful of users with the constructor's default score; the engine starts the input
        # rotation ahead of the router and hands over its padded capture batch.
        _decode("qwen3 5 tokens recovery-aware", _QWEN3, tokens=5, layers=4, padding=1,
                score="recovery-aware", prepare_input=True),
        # Eight users, router outputs in the types an engine's fused router gives.
        _decode("qwen3 8 tokens eager", _QWEN3, tokens=8, layers=4, ids64=True, weights16=True),
        # A GELU model of an odd width whose layers keep what passes a threshold, ragged batch.
        _decode("gelu threshold 19 tokens", hidden=1152, width=704, experts=64, top_k=6, rank=32,
                tokens=19, layers=4, retention=0.25, activation="gelu_tanh", threshold=True),
        # The decode batch of the 48-layer study.
        _decode("qwen3 32 tokens graph", _QWEN3, tokens=32, layers=2, graph=True),
        # The benchmark's batch.
        _decode("qwen3 64 tokens graph", _QWEN3, tokens=64, layers=2, graph=True),
        # A busy server in the default score, eager, a batch that is not a power of two.
        _decode("olmoe 100 tokens recovery-aware", _OLMOE, tokens=100, layers=1,
                score="recovery-aware"),
        # A large captured batch with heavy-tailed inputs and a skewed router, part of it padding.
        _decode("qwen3.5 256 tokens skewed", _QWEN35, tokens=256, layers=1, padding=13,
                graph=True),
        # The wide layer of the budget sweep at its middle batch.
        _decode("wide 32 tokens", _WIDE, tokens=32, layers=1, retention=0.125),
        # Its largest batch, largest budget and full sketch.
        _decode("wide 256 tokens full screen", _WIDE, tokens=256, layers=1, retention=0.25,
                screen_keep=1.0),
        # Model load: the sketch of one layer of the study's model.
        {"name": "sketch of a layer", "kind": "sketch", "hidden": 2048, "width": 768,
         "experts": 128},
    ]


def _log_int(rng, low: int, high: int, step: int = 1) -> int:
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(low, min(high, round(value / step) * step))


def draw(rng) -> dict:
    hidden = _log_int(rng, 1024, 4096, 128)
    width = _log_int(rng, 384, 1536, 16)
    experts = _log_int(rng, 32, 256)
    if experts * width * hidden > 128 * 1536 * 4096:  # no layer above the largest one
        experts = 128 * 1536 * 4096 // (width * hidden)
    if rng.random() < 0.08:
        return {"kind": "sketch", "hidden": hidden, "width": width, "experts": experts}
    tokens = _log_int(rng, 1, 256)
    top_k = rng.choice((4, 6, 8, 8))
    graph = rng.random() < 0.5
    case = {
        **_DECODE, "tokens": tokens,
        "layers": 6 if tokens <= 2 else 4 if tokens <= 16 else 2 if tokens <= 48 else 1,
        "hidden": hidden, "width": width, "experts": experts, "top_k": top_k,
        "rank": rng.choice((0, 16, 32, 64, 64, 128)),
        "retention": math.exp(rng.uniform(math.log(1 / 16), math.log(1 / 4))),
        "screen_keep": rng.choice((0.5, 0.625, 0.625, 0.75, 1.0)),
        "score": rng.choice(("point", "point", "recovery-aware")),
        "activation": rng.choice(("silu", "silu", "gelu_tanh")),
        "inputs": rng.choice(("normal", "outliers", "student_t")),
        "skewed": rng.random() < 0.3, "renormalize": rng.random() < 0.7,
        "threshold": rng.random() < 0.15,
        "padding": rng.randrange(0, 1 + tokens // 8) if graph else 0,
        "ids64": rng.random() < 0.5, "weights16": rng.random() < 0.3,
        "prepare_input": rng.random() < 0.25, "graph": graph,
    }
    # Keep a drawn step below the largest listed one, whatever was drawn together.
    most = _decode_work(listed()[-2])
    while case["tokens"] > 1 and any(
            a > b for a, b in zip(_decode_work(case).values(), most.values())):
        case["tokens"] //= 2
        case["padding"] = min(case["padding"], case["tokens"] // 8)
    return case


# -- preparation ------------------------------------------------------------------------
def _normal(shape: tuple[int, ...], sigma: float, generator: torch.Generator) -> torch.Tensor:
    out = torch.empty(shape, device="cuda", dtype=torch.bfloat16)
    return out.normal_(0.0, sigma, generator=generator)


def _plan(case: dict):
    return compile_budget(
        hidden_size=case["hidden"], expert_width=case["width"], top_k=case["top_k"],
        retention=case["retention"], screen_keep=case["screen_keep"],
    )


def _hidden_rows(case: dict, generator: torch.Generator) -> torch.Tensor:
    shape = (case["tokens"], case["hidden"])
    x = torch.randn(shape, device="cuda", generator=generator)
    if case["inputs"] == "student_t":  # three degrees of freedom, unit variance
        chi = torch.randn((*shape, 3), device="cuda", generator=generator).square().sum(-1)
        x = x / (chi / 3).sqrt() / math.sqrt(3.0)
    elif case["inputs"] == "outliers":  # one channel in a hundred is twenty times as large
        dims = torch.randperm(shape[1], device="cuda", generator=generator)
        x[:, dims[: math.ceil(0.01 * shape[1])]] *= 20.0
    return x.bfloat16()


def _route(case: dict, hidden: torch.Tensor, generator: torch.Generator):
    router = torch.randn((case["experts"], case["hidden"]), device="cuda", generator=generator)
    logits = hidden.float() @ (0.02 * router).T
    if case["skewed"]:
        logits = logits + torch.randn(case["experts"], device="cuda", generator=generator)
    weights, ids = torch.softmax(logits, dim=-1).topk(case["top_k"], dim=-1)
    if case["renormalize"]:
        weights = weights / weights.sum(-1, keepdim=True)
    ids = ids if case["ids64"] else ids.int()
    return ids.contiguous(), (weights.bfloat16() if case["weights16"] else weights).contiguous()


def _prepare_decode(case: dict, generator: torch.Generator) -> dict:
    plan = _plan(case)
    e, h, i, r = case["experts"], case["hidden"], case["width"], case["rank"]
    tokens = case["tokens"]
    device = torch.device("cuda", torch.cuda.current_device())
    workspace = ReaderWorkspace(plan, e, r, tokens, device)
    padding = None
    if case["padding"]:  # a captured batch is padded at its end
        padding = torch.arange(tokens, device="cuda") >= tokens - case["padding"]
    layers = []
    for _ in range(case["layers"]):
        gate_up = _normal((e, 2 * i, h), 0.02, generator)
        down = _normal((e, i, h), 0.02, generator).transpose(1, 2)  # channel-major
        encoder = decoder = None
        if r:  # a weight-only bank: an orthonormal U and U^T D of every expert
            basis = torch.randn((h, r), device="cuda", generator=generator)
            decoder = torch.linalg.qr(basis).Q.bfloat16()
            encoder = torch.matmul(decoder.T, down)
        hidden = _hidden_rows(case, generator)
        ids, weights = _route(case, hidden, generator)
        reader = ProgressiveReader(
            gate_up, down, encoder, decoder, plan, tokens, activation=case["activation"],
            selection_score=case["score"], workspace=workspace, sketch_builder="cuda",
            retain_reference_sketch=False,
            selection_threshold=0.0 if case["threshold"] else None,
        )
        if case["threshold"]:
            # The layer's threshold lets half of the cap through on average.
            reader(hidden, ids, weights, padding)
            scores = reader.scores[0][:tokens].flatten()
            reader.selection_threshold.copy_(
                scores.topk(max(1, tokens * plan.final_count // 2)).values[-1:])
            reader.read_work.zero_()
        layers.append((reader, hidden, ids, weights))
    state = {"layers": layers, "padding": padding, "early": case["prepare_input"]}
    # The kept channels of the last layer's live rows (the layers before it share the buffer).
    state["kept"] = layers[-1][0].candidate_ids[-1][: tokens - case["padding"]]
    if case["graph"]:
        _step(state)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _step(state)
        for reader, *_ in layers:
            reader.read_work.zero_()
        state.update(graph=graph, out=out)
    torch.cuda.synchronize()
    return state


def _step(state: dict) -> list[torch.Tensor]:
    """One decode step: every layer once; each layer's output rows."""
    out = []
    padding = state["padding"]
    for reader, hidden, ids, weights in state["layers"]:
        early = state["early"] and reader.prepare_input(hidden, padding)
        out.append(reader(hidden, ids, weights, padding, input_prepared=early))
    return out


def prepare(case: dict, seed: int) -> dict:
    generator = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "decode":
        return _prepare_decode(case, generator)
    shape = (case["experts"], 2 * case["width"], case["hidden"])
    return {
        "gate_up": _normal(shape, 0.02, generator),
        "signs": block_hadamard_signs(case["hidden"], "cuda"),
    }


def run(state: dict):
    if "gate_up" in state:
        return build_sketch_on_device(state["gate_up"], state["signs"])
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = _step(state)
    return {"out": out, "kept": state["kept"],
            "read_work": [reader.read_work for reader, *_ in state["layers"]]}


# -- what a pass cannot do without -------------------------------------------------------
def _decode_work(case: dict) -> dict:
    """Expected bytes and operations of a step, for tokens that route and keep independently.

    A routed expert's sketch and encoder rows and every native row that some token keeps are
    read once per layer; nothing is counted twice for tokens that share it.
    """
    plan = _plan(case)
    h, i, e, k, r = (case[x] for x in ("hidden", "width", "experts", "top_k", "rank"))
    t = case["tokens"] - case["padding"]
    n, keep, blocks = plan.candidate_count, plan.screen_coordinates, h // 128
    f = plan.final_count // 2 if case["threshold"] else plan.final_count
    kept = f / n
    routed = e * (1 - (1 - k / e) ** t)  # experts that some token routes to
    columns = e * i * (1 - (1 - kept * k / e) ** t)  # channels that some token keeps
    skipped = e * i * (1 - (1 - (1 - kept) * k / e) ** t)  # that some token skips
    coordinates = e * h * (1 - (1 - keep / 128 * k / e) ** t)  # sketch columns some token needs
    planes = 2 if case["score"] == "recovery-aware" else 1
    moved = (
        coordinates * i / 2  # two bits per trit of the 2 I rows
        + routed * blocks * planes * 4 * i + routed * i * (4 if planes == 1 else 12)
        + columns * 6 * h
        + skipped * 2 * r + 2 * h * r
        + case["tokens"] * (4 * h + k * ((8 if case["ids64"] else 4)
                                         + (2 if case["weights16"] else 4)))
    )
    operations = 2 * t * (2 * n * keep * blocks + 3 * f * h + (n - f) * r + h * r)
    return {"bytes": case["layers"] * moved, "flops": case["layers"] * operations}


def work(case: dict) -> dict:
    if case["kind"] == "decode":
        return _decode_work(case)
    weights = case["experts"] * 2 * case["width"] * case["hidden"]
    blocks = weights // 128
    # Two layouts of two bits per weight, scale and residual variance per block; seven
    # butterfly stages, the sign and scale products, and the three sums of the rule.
    return {"bytes": 2 * weights + 2 * weights / 4 + 4 * blocks + case["hidden"],
            "flops": 16 * weights}


def tolerance(case: dict) -> dict:
    if case["kind"] == "decode":
        return {"rel": 1e-2}  # BF16 outputs of the same kept channels
    # FP16 statistics; a coordinate within rounding of the ternary threshold may fall either way.
    return {"rel": 5e-4, "differ": 1e-5}
