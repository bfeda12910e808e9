"""Kernels at the sizes where their tiling can go wrong: remainders, smallest and largest."""

import pytest
import torch

import cases
from device import dispatch
from cfm_b200.reader.sketch import (
    block_hadamard_signs, build_sketch, build_sketch_on_device, repack_sketch,
    repack_sketch_grouped,
)
from helpers import prepared_case, relative_l2, run_oracle
from test_gpu_parity import make_reader, run_reader

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,width,hidden", [(1, 16, 128), (3, 48, 256), (2, 80, 1152)])
def test_sketch_builder_with_partial_row_tiles(experts, width, hidden):
    """A CTA of the builder takes 128 rows; 32, 96 and 160 rows leave warps without any."""
    device = torch.device("cuda:0")
    generator = torch.Generator().manual_seed(width)
    weights = (torch.randn(experts, 2 * width, hidden, generator=generator) * 0.02).bfloat16()
    weights[0, 3] = 0.0  # no coordinate above the threshold of a row of zeros
    weights = weights.to(device)
    signs = block_hadamard_signs(hidden, device)
    codes, statistics = build_sketch(weights, signs)
    words, grouped, fast = build_sketch_on_device(weights, signs)
    assert torch.equal(words, repack_sketch(codes, 2 * width, hidden))
    assert torch.equal(grouped, repack_sketch_grouped(codes, 2 * width, hidden))
    torch.testing.assert_close(fast.float(), statistics.float(), rtol=2e-3, atol=1e-7)


# hidden, width, experts, top_k, rank, tokens, retention, screen keep, activation, score, options
LAYERS = {
    # One warp of a tile per split of the blocks, an odd top_k, one block.
    "screen-one-block": (128, 48, 8, 3, 8, 1, 0.25, 0.5, "silu", "point", {}),
    # The tcgen05 screen at the edge of its 64 channels, passes of eight with a remainder.
    "tcgen05-ragged": (384, 80, 16, 2, 8, 9, 0.25, 0.5, "silu", "point", {"tensor_engine": "tcgen05"}),
    "tcgen05-risk-sixteen": (256, 80, 4, 2, 16, 35, 0.25, 1.0, "silu", "recovery-aware", {}),
    # Down columns: H not a multiple of 256, tiles per token and listed ones.
    "down-columns": (1152, 64, 8, 2, 32, 3, 0.5, 0.625, "silu", "point", {}),
    "down-listed": (1152, 208, 32, 3, 64, 8, 0.5, 0.625, "gelu_tanh", "point", {}),
    # Expert-major exact with the tiles per token: three tokens per expert and more, up to 16 / 3.
    "union-exact-only": (640, 112, 12, 3, 16, 18, 0.25, 0.625, "silu", "point", {}),
    # Twelve tokens and more, just below one token per expert and at it: exact rows by token, by pair.
    "exact-by-token": (384, 48, 64, 2, 16, 31, 0.3, 0.625, "silu", "point", {}),
    "exact-by-pair": (384, 48, 64, 2, 16, 32, 0.3, 0.625, "silu", "point", {}),
    # One step per quarter of the columns, fewer rows than a tile; a quarter that is no whole turn.
    "union-one-step": (128, 16, 4, 2, 8, 16, 0.25, 1.0, "silu", "point", {}),
    "union-part-turn": (640, 176, 6, 5, 128, 33, 0.3, 0.625, "gelu_tanh", "point", {}),
    # Several passes per expert.
    "union-risk": (512, 80, 4, 3, 256, 70, 0.2, 0.5, "silu", "recovery-aware", {}),
    # Expert-major down too: two column blocks of the encoder, an odd top_k, remainders everywhere.
    "union-down": (1280, 48, 64, 5, 128, 90, 0.3, 0.625, "gelu_tanh", "point", {}),
    # An eighth of a column block of the encoder.
    "union-down-risk": (1280, 80, 60, 3, 8, 110, 0.2, 0.5, "silu", "recovery-aware", {}),
    # More than eight slots, no recovery map, few rows.
    "union-down-many-slots": (1280, 16, 64, 12, 0, 64, 0.25, 0.625, "silu", "point", {}),
    # Requested below the sizes of the rule.
    "union-requested": (384, 96, 16, 2, 32, 8, 0.25, 0.625, "silu", "point",
                        {"row_engine": "expert_major"}),
}


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("name", LAYERS)
def test_layer_at_the_edges(oracle, name, padded):
    h, i, e, k, rank, tokens, retention, keep, activation, score, options = LAYERS[name]
    padding = [t % 5 == 1 for t in range(tokens)] if padded else None
    case = cases._random(name, h + i + tokens, h, i, e, k, rank, tokens, retention, keep, activation,
                         padding=padding, score=score)
    item = prepared_case(case)
    reader = make_reader(item, capacity=tokens + 3, **options)
    out = run_reader(reader, case).cpu()
    assert int(reader.workspace.status.abs().sum()) == 0
    own = dict(norms=reader.norms.cpu())
    if reader.recovery_geometry is not None:
        own["geometry"] = reader.recovery_geometry.cpu()
    want = run_oracle(oracle, item, **own)
    active = torch.ones(tokens, dtype=torch.bool) if case.padding is None else ~case.padding
    assert torch.equal(reader.partial[:tokens].cpu()[active], want["partial"][active])
    assert torch.equal(reader.scores[0][:tokens].cpu()[active], want["scores"][active])
    assert torch.equal(reader.candidate_ids[-1][:tokens].cpu()[active], want["candidate_ids"][active])
    torch.testing.assert_close(out.float()[active], want["output"][active], rtol=0.025, atol=0.02)
    exact = run_oracle(oracle, item, fp32=True, **own)
    assert relative_l2(out[active], exact["output"][active]) < 1e-2
    assert not out[~active].any()
    if rank:
        torch.testing.assert_close(reader.latent[:tokens].cpu()[active], want["latent"][active],
                                   rtol=0.015, atol=0.01)
        assert not reader.latent[:tokens].cpu()[~active].any()
    # Exact projections and activations of the kept channels, where the kernels leave them.
    lists = want["candidate_ids"].long()
    gathered = reader.activations[:tokens].cpu().reshape(tokens, -1).gather(1, lists.clamp_min(0))
    sums = reader.workspace.exact[:tokens].cpu()
    phi = torch.nn.functional.silu if activation == "silu" else (
        lambda x: torch.nn.functional.gelu(x, approximate="tanh"))
    feature = phi(sums[:, 0].bfloat16().float()).bfloat16().float() * sums[:, 1].bfloat16().float()
    mask = active[:, None] & (lists >= 0)
    torch.testing.assert_close(gathered.float()[mask], feature[mask], rtol=0.02, atol=1e-3)


@pytest.mark.parametrize("score", ["point", "recovery-aware"])
@pytest.mark.parametrize("tokens", [1, 5, 9, 17, 40])
@pytest.mark.parametrize("hidden,width", [(128, 16), (256, 112), (384, 128), (640, 144), (1152, 272)])
def test_tcgen05_screen_at_the_edges_of_its_tiles(oracle, hidden, width, tokens, score):
    """Channels around 128 per CTA and 32 per warp, blocks around the lengths of its rings, passes of
    four, eight and sixteen tokens with remainders: every projection and score of the oracle."""
    case = cases._random("tiles", hidden + tokens, hidden, width, 5, 2, 8, tokens, 0.25, 0.75, score=score)
    item = prepared_case(case)
    reader = make_reader(item, capacity=tokens, tensor_engine="tcgen05")
    run_reader(reader, case)
    assert int(reader.workspace.status.abs().sum()) == 0
    own = dict(norms=reader.norms.cpu())
    if reader.recovery_geometry is not None:
        own["geometry"] = reader.recovery_geometry.cpu()
    want = run_oracle(oracle, item, **own)
    assert torch.equal(reader.partial[:tokens].cpu(), want["partial"])
    assert torch.equal(reader.scores[0][:tokens].cpu(), want["scores"])


# 129 blocks: the products of a tile no longer fit shared memory, and a warp has a tile to itself.
@pytest.mark.parametrize("score", ["point", "recovery-aware"])
@pytest.mark.parametrize("hidden,width,experts,top_k,tokens", [
    (4096, 1536, 8, 8, 1), (4096, 1536, 8, 4, 9), (2048, 512, 32, 8, 4), (16384, 48, 3, 2, 5),
    (16512, 16, 3, 2, 1), (16512, 80, 4, 3, 11),
])
def test_the_two_expert_major_screens_agree(oracle, hidden, width, experts, top_k, tokens, score):
    """Warp-level and tcgen05 screen at sizes where a call by itself takes one of them only."""
    case = cases._random("screens", hidden + tokens, hidden, width, experts, top_k, 8, tokens, 0.25, 0.625,
                         score=score)
    item = prepared_case(case)
    want = None
    for engine in (1, 2):  # CFM_ENGINE_TCGEN05, CFM_ENGINE_WARP
        reader = make_reader(item, capacity=tokens)
        reader._layer.tensor_engine = engine
        run_reader(reader, case)
        reader.check_status()
        if want is None:
            own = dict(norms=reader.norms.cpu())
            if reader.recovery_geometry is not None:
                own["geometry"] = reader.recovery_geometry.cpu()
            want = run_oracle(oracle, item, **own)
        assert torch.equal(reader.partial[:tokens].cpu(), want["partial"])
        assert torch.equal(reader.scores[0][:tokens].cpu(), want["scores"])


def test_expert_major_stages_repeat_and_misaligned_output():
    """The stages on their own, twice, and an output that 16-byte stores cannot take."""
    case = cases._random("stages", 5, 1280, 48, 60, 3, 16, 112, 0.25, 0.625)
    reader = make_reader(prepared_case(case))
    whole = run_reader(reader, case).clone()
    device = whole.device
    hidden, ids, weights = (t.to(device) for t in (case.hidden, case.ids, case.weights))
    room = torch.zeros(whole.numel() + 1, dtype=whole.dtype, device=device)
    out = room[1:].view_as(whole)
    call = reader._call_struct(112, hidden, ids, weights, None, out, False)
    for stage in ("cfm_prepare_input", "cfm_route", "cfm_screen", "cfm_select", "cfm_exact", "cfm_exact",
                  "cfm_down", "cfm_down", "cfm_encode", "cfm_output"):
        reader._stage(stage, call)
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), whole.float(), rtol=0.016, atol=2e-3)


@pytest.mark.parametrize("width", [256, 512, 768, 1024, 1536, 2048])
def test_selection_at_every_number_of_keys_per_thread(width):
    """Largest sizes of the selection's six variants, with and without ties at the cut."""
    case = cases._random("select", width, 128, width, 8, 8, 0, 2, 0.125, 0.5)
    reader = make_reader(prepared_case(case))
    for levels in (0, 7):
        run_reader(reader, case)
        scores = reader.scores[0][:2]
        if levels:  # few distinct scores: most of the cut's are ties, kept in candidate order
            call = reader._call_struct(2, *(t.cuda() for t in (case.hidden, case.ids, case.weights)),
                                       None, torch.empty(2, 128, dtype=torch.bfloat16, device="cuda"), False)
            scores.copy_(torch.randint(1, levels, scores.shape, device="cuda").float())
            call.scores_ready = 1
            reader._stage("cfm_select", call)
        torch.cuda.synchronize()
        order = scores.sort(dim=1, descending=True, stable=True).indices[:, : case.plan.final_count]
        assert torch.equal(reader.candidate_ids[-1][:2].long(), order.sort(dim=1).values)


@pytest.mark.parametrize("width", [256, 768, 1536, 2048])
@pytest.mark.parametrize("kind", ["one-bin", "crowded-bin", "few-not-zero", "any-bits"])
def test_selection_by_bins(kind, width):
    """Keys that all fall into one bin of the selection, more of them in the cut's bin than one warp
    compares and than the list takes, fewer than are kept that differ from zero, and any 32 bits."""
    case = cases._random("bins", width, 128, width, 8, 8, 0, 2, 0.125, 0.5)
    reader = make_reader(prepared_case(case))
    run_reader(reader, case)
    scores = reader.scores[0][:2]
    n, f = scores.shape[1], case.plan.final_count
    g = torch.Generator().manual_seed(width)
    if kind == "one-bin":
        keys = 0x3F800000 + torch.randperm(0x3FFFF, generator=g)[: 2 * n].view(2, n)
    elif kind == "crowded-bin":  # some 60 or 200 keys about the cut share a bin
        keys = 0x3F800000 + (torch.randperm(n * 16, generator=g)[: 2 * n] * (0x40000 // (60 * 16 * (1 + 2 * (width > 768))))).view(2, n)
    elif kind == "few-not-zero":
        keys = torch.where(torch.rand(2, n, generator=g) < 0.5 * f / n, 0x3F800000 + torch.arange(n), 0)
    else:
        keys = torch.randint(0, 1 << 32, (2, n), generator=g)
        keys[:, ::3] = keys[:, ::3] % 5 + 0xFFFFFFF0
    signed = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).int()
    scores.view(torch.int32).copy_(signed)
    call = reader._call_struct(2, *(t.cuda() for t in (case.hidden, case.ids, case.weights)), None,
                               torch.empty(2, 128, dtype=torch.bfloat16, device="cuda"), False)
    call.scores_ready = 1
    reader._stage("cfm_select", call)
    torch.cuda.synchronize()
    kept = keys.sort(dim=1, descending=True, stable=True).indices[:, :f].sort(dim=1).values
    assert torch.equal(reader.candidate_ids[-1][:2].cpu().long(), kept)
    mask = torch.zeros(2, n, dtype=torch.uint8).scatter_(1, kept, 1)
    assert torch.equal(reader.workspace.selected[:2].cpu().view(2, n).to(torch.uint8), mask)


@pytest.mark.parametrize("rank,width,tokens", [(8, 400, 26), (64, 272, 40), (256, 256, 42)])
def test_encoder_rows_shared_by_an_experts_pairs(rank, width, tokens):
    """Large calls sum the encoder for several pairs of an expert at a time; the stage on its own takes a
    pair at a time.  The same latents, with padding and with passes that are not full."""
    _shared_encoder(rank, width, tokens, experts=6, top_k=5, passes=16)


@pytest.mark.parametrize("rank,width,tokens,experts,passes", [
    (64, 176, 48, 60, 4),   # four pairs per expert: the rule's edge, one part per pass
    (16, 272, 33, 20, 8),
    (128, 176, 50, 16, 8),  # just below sixteen
])
def test_encoder_rows_shared_by_fewer_pairs(rank, width, tokens, experts, passes):
    """The same in passes of four and eight pairs, with some experts' load far above the others'."""
    generator = torch.Generator().manual_seed(experts)
    load = 1.0 / (3.0 + torch.arange(experts))
    routes = torch.multinomial(load.expand(tokens, -1), 5, generator=generator).tolist()
    _shared_encoder(rank, width, tokens, experts=experts, top_k=5, passes=passes, routes=routes)


def _shared_encoder(rank, width, tokens, experts, top_k, passes, routes=None):
    hidden = 4096
    case = cases._random("shared", rank, hidden, width, experts, top_k, rank, tokens, 0.7, 0.625,
                         routes=routes, padding=[t % 7 == 3 for t in range(tokens)])
    took = dispatch(tokens, hidden=hidden, width=width, experts=experts, top_k=top_k, rank=rank,
                    final_count=case.plan.final_count)
    assert took["shares_encoder"] and took["pass_pairs"] == passes
    reader = make_reader(prepared_case(case))
    run_reader(reader, case)
    device = reader.latent.device
    whole = reader.latent[:tokens].clone()
    assert whole.abs().sum() > 0
    reader.latent.fill_(float("nan"))
    call = reader._call_struct(tokens, *(t.to(device) for t in (case.hidden, case.ids, case.weights, case.padding)),
                               torch.empty(tokens, hidden, dtype=torch.bfloat16, device=device), False)
    reader._stage("cfm_encode", call)
    torch.cuda.synchronize()
    assert torch.equal(whole, reader.latent[:tokens])
