"""The rules that pick a call's kernels, on the host."""

import pytest

import device

QWEN3 = dict(hidden=2048, width=768, experts=128, top_k=8, final_count=756, rank=64)
OLMOE = dict(QWEN3, width=1024, experts=64, final_count=1008)
WIDE = dict(QWEN3, hidden=4096, width=1536, final_count=1536, rank=128)
SMALL = dict(QWEN3, width=512, experts=256, final_count=504)


@pytest.mark.parametrize("ranks", [2, 4, 8])
@pytest.mark.parametrize("layer", [QWEN3, OLMOE, WIDE, SMALL])
def test_a_rank_takes_the_passes_of_one_gpu(layer, ranks):
    """Passes are chosen by tokens per expert, which sharing the experts does not change."""
    share = dict(layer, experts=layer["experts"] // ranks, global_experts=layer["experts"],
                 tensor_engine=1)
    whole = dict(layer, tensor_engine=1)
    for tokens in (1, 4, 16, 32, 64, 100, 128, 256):
        assert device.dispatch(tokens, **share)["pass_pairs"] == device.dispatch(tokens, **whole)["pass_pairs"], tokens


@pytest.mark.parametrize("layer,ranks,tokens,tcgen05,pairs", [
    # Kernel times of one rank of `ranks`, us: the rule's kernel first.
    (QWEN3, 8, 16, 0, 8),    # 7.2; passes of four 12.5, of eight 14.5
    (QWEN3, 8, 32, 0, 8),    # 12.8; passes of four 13.2, of sixteen 17.4
    (QWEN3, 8, 128, 1, 8),   # 18.9; of four 20.3, of sixteen 25.0, without 22.5
    (QWEN3, 2, 32, 1, 4),    # 20.3; of eight 22.1, without 32.8
    (SMALL, 8, 16, 0, 8),    # 7.3; of four 11.7
    (SMALL, 8, 64, 1, 4),    # 13.9; of sixteen 18.1, without 16.1
    (SMALL, 8, 256, 1, 8),   # 24.7; of sixteen 27.3
    (WIDE, 8, 32, 1, 4),     # 24.4; of sixteen 30.7, without 34.6
    (WIDE, 8, 256, 1, 16),   # 54.3; of eight 63.0
])
def test_screen_of_a_rank(layer, ranks, tokens, tcgen05, pairs):
    share = dict(layer, experts=layer["experts"] // ranks, global_experts=layer["experts"])
    took = device.dispatch(tokens, **share)
    assert (took["tcgen05"], took["pass_pairs"]) == (tcgen05, pairs)


@pytest.mark.parametrize("layer,tokens,by_pair", [
    (QWEN3, 12, 0), (QWEN3, 15, 0), (QWEN3, 16, 1), (OLMOE, 8, 0), (OLMOE, 11, 0), (OLMOE, 12, 1),
    (SMALL, 31, 0), (SMALL, 32, 1), (WIDE, 32, 1),
])
def test_exact_rows_by_pair_from_one_token_per_expert_on(layer, tokens, by_pair):
    assert device.dispatch(tokens, **layer)["by_pair"] == by_pair


@pytest.mark.parametrize("tokens", [8, 12, 64])
def test_a_rank_walks_pairs_from_eight_tokens_on(tokens):
    share = dict(SMALL, experts=SMALL["experts"] // 8, global_experts=SMALL["experts"])
    assert device.dispatch(tokens, **share)["by_pair"]
