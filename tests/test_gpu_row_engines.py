"""The expert-major kernels of the native rows against the gathers per token: the same layer and calls
through `row_engine="auto"` (unions of an expert's kept rows where the sizes call for them) and
`"per_token"`."""

import pytest
import torch

import cases
from helpers import prepared_case, run_oracle
from test_gpu_parity import make_reader

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
