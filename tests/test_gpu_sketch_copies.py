"""What a reader keeps of its sketch: the row-major copy, and the others only where they are wanted."""

import ctypes

import pytest
import torch

from cfm_b200.reader.progressive import ProgressiveReader
from helpers import prepared
from test_gpu_parity import make_reader, run_reader

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["qwen35-e16-t4", "gh-full", "olmoe-t1"])
@pytest.mark.parametrize("builder", ["given", "cuda"])
def test_calls_read_the_row_major_copy_only(name, builder):
    item = prepared(name)
    case = item["case"]
    if builder == "given":
        both, lean = make_reader(item), make_reader(item, retain_reference_sketch=False)
    else:
        gate_up, down = case.gate_up.cuda(), item["down"].transpose(1, 2).contiguous().cuda().transpose(1, 2)
        bank = [t.cuda() if t is not None else None for t in (case.encoder, case.decoder)]
        both, lean = (ProgressiveReader(gate_up, down, *bank, case.plan, case.hidden.shape[0], sketch_builder="cuda",
                                        activation=case.activation, selection_score=case.score, **kept)
                      for kept in ({}, {"retain_reference_sketch": False}))
    want, out = run_reader(both, case), run_reader(lean, case)
    assert torch.equal(out, want)
    assert lean.sketch_codes is None and lean.sketch_words is None and lean._layer.sketch is None
    copy = both.sketch_words.numel() * 4
    assert copy == both.sketch_grouped_words.numel() * 4
    assert both.sketch_resident_bytes - lean.sketch_resident_bytes == copy


def test_a_layer_without_any_sketch_is_refused():
    item = prepared("tiny")
    reader = make_reader(item, retain_reference_sketch=False, retain_coordinate_sketch=True)
    assert reader.sketch_codes is None and reader.sketch_words is not None
    grouped = reader._layer.sketch_grouped
    want = run_reader(reader, item["case"]).clone()
    reader._layer.sketch_grouped = None  # the coordinate-major copy serves alone, and in place of a misaligned one
    assert torch.equal(run_reader(reader, item["case"]), want)
    reader._layer.sketch_grouped = grouped + 4
    assert torch.equal(run_reader(reader, item["case"]), want)
    reader._layer.sketch = None
    call = reader._call_struct(1, *(t.cuda() for t in (item["case"].hidden, item["case"].ids, item["case"].weights)),
                               None, want, False)
    code = reader._library.cfm_reader_forward(
        reader._layer_ref, reader._workspace_pointer, reader._workspace_capacity, ctypes.byref(call), None)
    assert code == -1
