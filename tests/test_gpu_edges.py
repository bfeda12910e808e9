"""Kernels at the sizes where their tiling can go wrong: remainders, smallest and largest."""

import pytest
import torch

from cfm_b200.reader.sketch import (
    block_hadamard_signs, build_sketch, build_sketch_on_device, repack_sketch,
    repack_sketch_grouped,
)

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
