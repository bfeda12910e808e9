"""The screen of one expert-parallel rank: most of a call's (token, expert) pairs are another rank's."""

import socket
from contextlib import contextmanager

import pytest
import torch
import torch.distributed as dist

import cases
from cfm_b200.reader.progressive import ProgressiveReader
from helpers import prepared_case, run_oracle
from test_gpu_parity import _channel_major, _move_statistics

pytestmark = pytest.mark.gpu


@contextmanager
def one_rank():
    with socket.socket() as sock:
        sock.bind(("127.0.0.1", 0))
        port = sock.getsockname()[1]
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1)
    try:
        yield
    finally:
        dist.destroy_process_group()


def _expert_map(held: int, experts: int) -> torch.Tensor:
    """The first `held` of the experts are this rank's."""
    return torch.tensor([e if e < held else -1 for e in range(experts)], dtype=torch.int32)


def _screen(reader, tokens, hidden, ids, weights, padding=None):
    out = torch.empty(tokens, hidden.shape[1], dtype=torch.bfloat16, device="cuda")
    call = reader._call_struct(tokens, hidden, ids, weights, padding, out, False)
    for stage in ("cfm_prepare_input", "cfm_route", "cfm_screen"):
        reader._stage(stage, call)
    return call, out


# Fewer pairs than a row of CTAs clears, several rows of them, and more pairs than all rows take at a time;
# widths of one CTA of the tcgen05 screen, of a part of one, and of several.
@pytest.mark.parametrize("engine", ["mma_sync", "tcgen05"])
@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("width,tokens", [(16, 2), (16, 37), (16, 171), (128, 9), (272, 40)])
def test_projections_of_dead_pairs_are_zero(oracle, width, tokens, padded, engine):
    held, experts, top_k = 3, 13, 4
    generator = torch.Generator().manual_seed(width + tokens)
    routes = [torch.randperm(experts, generator=generator)[:top_k].tolist() for _ in range(tokens)]
    padding = [t % 3 == 1 for t in range(tokens)] if padded else None
    case = cases._random("dead", width + tokens, 256, width, held, top_k, 0, tokens, 0.25, 0.625,
                         routes=routes, padding=padding)
    item = prepared_case(case)
    placement = _expert_map(held, experts)
    with one_rank():
        reader = ProgressiveReader(
            case.gate_up.cuda(), _channel_major(item["down"], "cuda"), None, None, case.plan, tokens,
            expert_map=placement, recovery_owner=True, tensor_engine=engine,
            sketch=(item["codes"].cuda(), _move_statistics(item["statistics"], "cuda")))
    reader.partial.fill_(float("nan"))
    _screen(reader, tokens, case.hidden.cuda(), case.ids.cuda(), case.weights.cuda(),
            case.padding.cuda() if padded else None)
    torch.cuda.synchronize()
    want = run_oracle(oracle, item, expert_map=placement, norms=reader.norms.cpu())
    assert int(reader.workspace.status.abs().sum()) == 0
    got = reader.partial[:tokens].cpu().view(tokens, 2, top_k, width)
    local = reader.ids[:tokens].cpu() >= 0
    if padded:
        local &= ~case.padding[:, None]
    dead = ~local[:, None, :, None].expand_as(got)
    assert dead.any() and not got[dead].any()
    assert torch.equal(got[~dead], want["partial"].view_as(got)[~dead])


def test_a_rank_screens_its_share_faster_than_one_gpu_screens_all():
    """An eighth of the pairs of 256 tokens against all of them.  (The margin is wide: 28 us against 76, and
    with all dead pairs cleared by the CTAs of one row the share took 409.)"""
    hidden, width, experts, held, top_k, tokens = 2048, 768, 128, 16, 8, 256
    plan = cases._plan(hidden, width, top_k, 0.123046875, 0.625)
    generator = torch.Generator(device="cuda").manual_seed(1)

    def normal(*shape):
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=generator)

    gate_up, down = normal(experts, 2 * width, hidden), normal(experts, width, hidden)
    x = torch.randn(tokens, hidden, device="cuda", generator=generator).bfloat16()
    ids = torch.rand(tokens, experts, device="cuda", generator=generator).argsort(1)[:, :top_k].int().contiguous()
    weights = torch.full((tokens, top_k), 1.0 / top_k, device="cuda")
    options = dict(sketch_builder="cuda", retain_reference_sketch=False, selection_score="point")
    whole = ProgressiveReader(gate_up, down.transpose(1, 2), None, None, plan, tokens, **options)
    with one_rank():
        share = ProgressiveReader(gate_up[:held], down[:held].transpose(1, 2), None, None, plan, tokens,
                                  expert_map=_expert_map(held, experts), recovery_owner=True, **options)
    times = []
    for reader in (whole, share):
        call, keep = _screen(reader, tokens, x, ids, weights)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        for timed in (False, True):
            start.record()
            for _ in range(50):
                reader._stage("cfm_screen", call)
            end.record()
            torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    assert times[1] < times[0], times
