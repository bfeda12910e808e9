"""The expert-major kernels of the native rows against the gathers per token: the same layer and calls
through `row_engine="auto"` (unions of an expert's kept rows where the sizes call for them) and
`"per_token"`."""

import pytest
import torch

import cases
from cfm_b200.reader.budget import compile_budget
from cfm_b200.reader.progressive import ProgressiveReader
from helpers import prepared_case, run_oracle
from test_gpu_edges import LAYERS
from test_gpu_parity import make_reader, run_reader

pytestmark = pytest.mark.gpu


def _batch(case, tokens, seed, busiest=None, padded=False):
    """Inputs of another call on the layer of `case`; with `busiest` every token goes to the first experts."""
    g = torch.Generator().manual_seed(seed)
    h, e, k = case.plan.hidden_size, case.gate_up.shape[0], case.plan.top_k
    hidden = torch.randn(tokens, h, generator=g).bfloat16()
    ids = torch.stack([torch.randperm(busiest or e, generator=g)[:k] for _ in range(tokens)]).int()
    weights = torch.rand(tokens, k, generator=g) * 0.6 + 0.2
    padding = (torch.arange(tokens) % 4 == 1) if padded else None
    return hidden, ids, weights, padding


# hidden, width, experts, top_k, rank: gathers of the down rows, and the expert-major down kernel.
@pytest.mark.parametrize("shape", [(384, 48, 12, 3, 16), (1280, 48, 64, 5, 128)])
def test_unscreened_calls_that_change_their_routes(oracle, shape):
    """A plan that keeps everything has no screen between the grouping and the selection; calls of
    different length, routing and padding follow one another on one workspace without a pause."""
    h, i, e, k, rank = shape
    case = cases._random("unscreened", 31, h, i, e, k, rank, 8 * e, 1.0, 1.0)
    assert case.plan.final_count == case.plan.candidate_count
    item = prepared_case(case)
    reader = make_reader(item)
    plain = make_reader(item, row_engine="per_token")
    calls = [_batch(case, tokens, seed, busiest, padded) for seed, (tokens, busiest, padded) in enumerate(
        [(4 * e, None, False), (3 * e // 2, 2 * k, True), (8 * e, None, True), (e, k, False), (2 * e, None, False)])]
    device = [tuple(x.cuda() if x is not None else None for x in call) for call in calls]
    outs = [reader(*call) for call in device]
    wants = [plain(*call) for call in device]
    torch.cuda.synchronize()
    for out, want in zip(outs, wants):
        torch.testing.assert_close(out.float(), want.float(), rtol=0.016, atol=2e-3)
    hidden, ids, weights, padding = calls[1]
    case.hidden, case.ids, case.weights, case.padding = hidden, ids, weights, padding
    want = run_oracle(oracle, item, norms=reader.norms.cpu())
    torch.testing.assert_close(outs[1].cpu().float(), want["output"], rtol=0.025, atol=0.02)


def _layer(experts, hidden, width, top_k, rank, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    gate_up = torch.empty(experts, 2 * width, hidden, device="cuda", dtype=torch.bfloat16).normal_(0, 0.02, generator=g)
    down = torch.empty(experts, width, hidden, device="cuda", dtype=torch.bfloat16).normal_(0, 0.02, generator=g)
    down = down.transpose(1, 2)
    if not rank:
        return gate_up, down, None, None
    decoder = torch.linalg.qr(torch.randn(hidden, rank, device="cuda", generator=g)).Q.bfloat16()
    return gate_up, down, torch.matmul(decoder.T, down), decoder


def _inputs(kind, tokens, hidden, experts, top_k, seed):
    """Hidden rows and routes; outliers: one column in a hundred is twenty times as large."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(tokens, hidden, device="cuda", generator=g)
    if kind == "outliers":
        x[:, torch.randperm(hidden, device="cuda", generator=g)[: hidden // 100]] *= 20
    elif kind == "student_t":
        x /= (torch.randn(tokens, hidden, 3, device="cuda", generator=g).square().sum(-1) / 3).sqrt()
    ids = torch.rand(tokens, experts, device="cuda", generator=g).topk(top_k, dim=1).indices.int().contiguous()
    weights = torch.rand(tokens, top_k, device="cuda", generator=g) * 0.6 + 0.2
    return x.bfloat16(), ids, weights


def _readers(layer, plan, tokens, engine="auto"):
    return [ProgressiveReader(*layer, plan, tokens, selection_score="point", sketch_builder="cuda",
                              retain_reference_sketch=False, row_engine=which) for which in (engine, "per_token")]


def _plan(name):
    h, i, e, k, _, _, retention = WIDE[name]
    return compile_budget(hidden_size=h, expert_width=i, top_k=k, retention=retention,
                          screen_keep=1.0 if retention == 1.0 else 0.625)


# hidden, width, experts, top_k, rank, tokens, retention
WIDE = {
    "kept-256": (2048, 768, 40, 8, 64, 256, 1.0),
    "kept-1024": (2048, 768, 40, 8, 64, 1024, 1.0),
    "screened-96": (2048, 512, 40, 8, 64, 96, 0.125),
    "screened-200": (4096, 320, 24, 6, 128, 200, 0.25),
    "screened-130": (1152, 208, 66, 5, 16, 130, 0.2),
}


@pytest.mark.parametrize("inputs", ["normal", "outliers", "student_t"])
@pytest.mark.parametrize("name", WIDE)
def test_activations_are_those_of_the_gathers(name, inputs):
    """Bit by bit, however many sums of a CTA are in doubt, and again in every call."""
    h, i, e, k, rank, tokens, _ = WIDE[name]
    reader, plain = _readers(_layer(e, h, i, k, rank), _plan(name), tokens)
    call = _inputs(inputs, tokens, h, e, k, 7)

    def kept(r):
        lists = r.candidate_ids[-1][:tokens].long()
        return r.activations[:tokens].view(tokens, -1).gather(1, lists.clamp_min(0)).view(torch.int16)

    plain(*call)
    want = kept(plain)
    first = reader(*call)
    assert torch.equal(reader.candidate_ids[-1][:tokens], plain.candidate_ids[-1][:tokens])
    sums = reader.workspace.exact.clone()
    for _ in range(10):
        assert torch.equal(kept(reader), want)
        reader.activations.zero_()
        assert torch.equal(reader(*call), first)
    assert torch.equal(reader.workspace.exact, sums)


def test_down_sums_are_as_near_to_64_bits_as_the_gathers():
    """Shares of the expert sums that round to another BF16 value than the sum in 64 bits does.  The
    gathers add at most sixteen terms in a row in FP32 and turn 90 of the 786,432; the tensor cores,
    which truncate, turn as many when a sum leaves them every 64 rows, and 819 in one chain of 1536."""
    h, i, e, k, tokens = 2048, 1536, 40, 4, 96
    plan = compile_budget(hidden_size=h, expert_width=i, top_k=k, retention=1.0, screen_keep=1.0)
    layer = _layer(e, h, i, k, 0)
    reader, plain = _readers(layer, plan, tokens, "expert_major")
    call = _inputs("normal", tokens, h, e, k, 11)
    reader(*call)
    plain(*call)
    assert torch.equal(reader.activations, plain.activations)
    sums = torch.zeros(tokens, k, h, device="cuda")
    for tile in plain.down_parts.view(tokens, -1, h)[:, : k * i // 64].reshape(tokens, k, -1, h).unbind(2):
        sums += tile
    union = reader.down_parts.view(-1).view(torch.bfloat16)[: tokens * k * h].view(tokens, k, h)
    wrong = torch.zeros(2, dtype=torch.int64, device="cuda")
    for t in range(tokens):
        down = layer[1].transpose(1, 2)[reader.ids[t].long()].double()  # [K, I, H]
        want = torch.matmul(reader.activations[t].view(k, 1, i).double(), down)[:, 0]
        want = want.bfloat16()
        wrong += torch.stack([(sums[t].bfloat16() != want).sum(), (union[t] != want).sum()])
    gathers, unions = wrong.tolist()
    assert 0 < gathers and unions <= 2 * gathers


@pytest.mark.parametrize("inputs", ["normal", "outliers", "student_t"])
@pytest.mark.parametrize("name", WIDE)
def test_outputs_do_not_depend_on_the_batch(name, inputs):
    """Bit by bit: the gathers per token, the unions of the whole batch, and tokens on their own."""
    h, i, e, k, rank, tokens, _ = WIDE[name]
    reader, plain = _readers(_layer(e, h, i, k, rank), _plan(name), tokens)
    call = _inputs(inputs, tokens, h, e, k, 13)
    want, latent = plain(*call), plain.latent[:tokens].clone()
    out = reader(*call)
    assert torch.equal(out, want)
    if rank:
        assert torch.equal(reader.latent[:tokens], latent)
    for first, count in ((0, 1), (tokens - 1, 1), (tokens // 3, 9), (5, tokens // 2), (tokens // 2, tokens // 3)):
        part = reader(*(x[first : first + count] for x in call))
        assert torch.equal(part, want[first : first + count])


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("name", [n for n in LAYERS if n.startswith("union")])
def test_outputs_at_the_edges_are_those_of_the_gathers(name, padded):
    h, i, e, k, rank, tokens, retention, keep, activation, score, _ = LAYERS[name]
    padding = [t % 5 == 1 for t in range(tokens)] if padded else None
    item = prepared_case(cases._random(name, h + i + tokens, h, i, e, k, rank, tokens, retention, keep, activation,
                                       padding=padding, score=score))
    unions, plain = (make_reader(item, row_engine=engine) for engine in ("auto", "per_token"))
    want, out = run_reader(plain, item["case"]), run_reader(unions, item["case"])
    assert torch.equal(out, want)
    if rank:
        assert torch.equal(unions.latent[:tokens], plain.latent[:tokens])


@pytest.mark.parametrize("name", ["kept-256", "screened-96"])
def test_expert_major_down_sums(name):
    """On request the down and encoder rows are read expert-major too: the same bits in every call, those
    of the gathers but for roundings that the order of summation turns."""
    h, i, e, k, rank, tokens, _ = WIDE[name]
    reader, plain = _readers(_layer(e, h, i, k, rank), _plan(name), tokens, "expert_major")
    call = _inputs("outliers", tokens, h, e, k, 19)
    claims = 4  # of `work_counts`: pieces the expert-major down kernel has claimed
    want = plain(*call)
    assert plain.workspace.work_counts[claims] == 0
    first = reader(*call)
    assert reader.workspace.work_counts[claims] > 0
    torch.testing.assert_close(first.float(), want.float(), rtol=0.016, atol=2e-3)
    for _ in range(10):
        assert torch.equal(reader(*call), first)


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("name", [n for n in LAYERS if n.startswith("union-down")])
def test_expert_major_down_at_the_edges(name, padded):
    """The whole call, and its stages on their own, twice where they claim their work."""
    h, i, e, k, rank, tokens, retention, keep, activation, score, _ = LAYERS[name]
    padding = [t % 5 == 1 for t in range(tokens)] if padded else None
    item = prepared_case(cases._random(name, h + i + tokens, h, i, e, k, rank, tokens, retention, keep, activation,
                                       padding=padding, score=score))
    case = item["case"]
    unions, plain = (make_reader(item, row_engine=engine) for engine in ("expert_major", "per_token"))
    want, out = run_reader(plain, case), run_reader(unions, case).clone()
    assert unions.workspace.work_counts[4] > 0
    torch.testing.assert_close(out.float(), want.float(), rtol=0.016, atol=2e-3)
    device = [x.cuda() if x is not None else None for x in (case.hidden, case.ids, case.weights, case.padding)]
    again = torch.empty_like(out)
    call = unions._call_struct(tokens, *device, again, False)
    for stage in ("cfm_prepare_input", "cfm_route", "cfm_screen", "cfm_select", "cfm_exact", "cfm_down", "cfm_down",
                  "cfm_encode", "cfm_output"):
        unions._stage(stage, call)
    torch.cuda.synchronize()
    torch.testing.assert_close(again.float(), want.float(), rtol=0.016, atol=2e-3)


@pytest.mark.parametrize("engine", ["auto", "expert_major"])
def test_a_row_that_is_not_finite_reaches_only_tokens_that_kept_it(engine):
    h, i, e, k, rank, tokens, _ = WIDE["screened-96"]
    layer = _layer(e, h, i, k, rank)
    reader, plain = _readers(layer, _plan("screened-96"), tokens, engine)
    call = _inputs("normal", tokens, h, e, k, 17)
    reader(*call)
    chosen = reader.candidate_ids[-1][0, 0].item()  # a channel the first token keeps
    expert, channel = reader.ids[0, chosen // i].item(), chosen % i
    layer[1][expert, :, channel] = float("inf")  # the native weights are read in place
    out, want = reader(*call), plain(*call)
    keeps = ((reader.ids[:tokens] == expert)[:, :, None] & reader.selected[:tokens].view(tokens, k, i))[:, :, channel]
    assert keeps.any() and not keeps.any(1).all()
    assert out[~keeps.any(1)].isfinite().all() and not out[keeps.any(1)].isfinite().any()
    assert torch.equal(out.isnan(), want.isnan())
    torch.testing.assert_close(out.float().nan_to_num(), want.float().nan_to_num(), rtol=0.016, atol=2e-3)


# hidden, width, experts, top_k, rank, tokens: no map, an eighth of 64 latent columns, the largest rank
# with a remainder of three tokens, more slots than are on their way at a time.
@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("shape", [(4096, 16, 20, 5, 0, 80), (4096, 48, 20, 5, 8, 75), (2048, 32, 16, 3, 256, 147),
                                   (2048, 208, 30, 12, 32, 150)])
def test_output_of_sixteen_tokens_at_the_edges(shape, padded):
    h, i, e, k, rank, tokens = shape
    padding = [t % 7 == 3 or t >= tokens - 2 for t in range(tokens)] if padded else None
    item = prepared_case(cases._random("mix", h + i, h, i, e, k, rank, tokens, 0.4, 0.5, padding=padding))
    sixteen, one = (make_reader(item, row_engine=engine) for engine in ("auto", "per_token"))
    want, out = run_reader(one, item["case"]), run_reader(sixteen, item["case"])
    assert torch.equal(out, want)
    if rank:
        assert torch.equal(sixteen.latent[:tokens], one.latent[:tokens])
