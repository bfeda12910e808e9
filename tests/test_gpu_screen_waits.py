"""Waits of the tcgen05 screen that run out: a status, no half-summed projections, a context that goes on."""

import pytest
import torch

import cases
import device
from helpers import prepared_case, run_oracle
from test_gpu_parity import make_reader, run_reader

pytestmark = pytest.mark.gpu


# Passes of four, eight and sixteen tokens.
@pytest.mark.parametrize("score", ["point", "recovery-aware"])
@pytest.mark.parametrize("tokens", [5, 17, 40])
@pytest.mark.parametrize("hidden,width", [(128, 16), (1152, 272), (4096, 144)])
def test_waits_that_run_out_leave_no_wrong_projection(oracle, hidden, width, tokens, score):
    case = cases._random("waits", hidden + tokens, hidden, width, 5, 2, 8, tokens, 0.25, 0.75, score=score)
    item = prepared_case(case)
    reader = make_reader(item, capacity=tokens, tensor_engine="tcgen05")
    run_reader(reader, case)
    reader.check_status()
    own = dict(norms=reader.norms.cpu())
    if reader.recovery_geometry is not None:
        own["geometry"] = reader.recovery_geometry.cpu()
    want = run_oracle(oracle, item, **own)

    screen, status = device.impatient_screen(), reader.workspace.status
    inputs = [t.cuda() for t in (case.hidden, case.ids, case.weights)]
    call = reader._call_struct(tokens, *inputs, None, torch.empty_like(inputs[0]), False)
    gave_up = 0
    for _ in range(8):
        status.zero_()
        reader.partial.fill_(float("nan"))
        reader.scores[0].fill_(float("nan"))
        reader._enqueue(screen, "cfm_screen", call)
        torch.cuda.synchronize()
        for got, right in ((reader.partial, want["partial"]), (reader.scores[0], want["scores"])):
            got = got[:tokens].cpu()
            unwritten = got.isnan()
            assert torch.equal(got[~unwritten], right[~unwritten])
            assert int(status.abs().sum()) or not unwritten.any()
        gave_up += int(status.abs().sum())
    assert gave_up
    with pytest.raises(RuntimeError, match="status"):
        status.fill_(1)
        reader.check_status()

    status.zero_()
    run_reader(reader, case)
    reader.check_status()
    assert torch.equal(reader.partial[:tokens].cpu(), want["partial"])
    assert torch.equal(reader.scores[0][:tokens].cpu(), want["scores"])
