"""Prefill attention where a CTA has a pair of query tiles to itself: steps with pairs enough for the GPU."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import workloads
from oracle import hot_path
from test_prefill_attention_gpu import ATOL, _run
from test_sink_attention_gpu import Case

pytestmark = pytest.mark.gpu

# heads, kv_heads, dim, vdim.  Eight prompts of 900 tokens behind 40 cached ones are at least 96 pairs, which are not shared by
# a cluster, and with 40 cached tokens the two query tiles of a pair end in different K/V tiles.
LENGTHS, CHUNKS = [940] * 8, [900] * 8
# Keys narrower than the output rows, which are staged where the queries were: of one and two query heads a key/value head,
# and with two passes over the values.
NARROW_KEYS = [(4, 4, 64, 128), (4, 2, 64, 128), (2, 2, 40, 200)]


@pytest.mark.parametrize("window", [None, 300])
@pytest.mark.parametrize("sizes", NARROW_KEYS, ids=str)
def test_narrow_keys(sizes, window, device):
    case = Case(LENGTHS, CHUNKS, *sizes, window, 16, torch.bfloat16, seed=31)
    for _ in range(3):
        case.prefill(device)
        case.check()


# Keys that leave shared memory for one K stage: three and four 64-dim groups, one and two query heads a key/value head.
WIDE_KEYS = [(3, 3, 192, 128), (4, 2, 192, 128), (3, 3, 256, 256)]


@pytest.mark.parametrize("window", [None, 300])
@pytest.mark.parametrize("sizes", WIDE_KEYS, ids=str)
def test_wide_keys(sizes, window, device):
    """The last K/V tile of a pair is seen by its second query tile alone."""

    case = Case(LENGTHS, CHUNKS, *sizes, window, 16, torch.bfloat16, seed=32)
    for _ in range(3):
        case.prefill(device)
        case.check()


# One query tile, shared by eight ranks; 79 pairs, not shared.
@pytest.mark.parametrize("chunk,heads,kv_heads", [(20, 8, 2), (2500, 8, 1)])
def test_more_than_64k_cached_tokens(chunk, heads, kv_heads, device, status_clean):
    """The first and the last rows of the chunk; queries of three units, so that a few keys have most of the weight."""

    case = workloads.prefill_case(seed=33, prefix_lengths=(66_000,), chunk_lengths=(chunk,), q_heads=heads,
                                  kv_heads=kv_heads)
    case.query.mul_(3.0)
    _, out = _run(case, device)
    keys, values = case.key_blocks.clone(), case.value_blocks.clone()
    hot_path.write_packed_kv(case.new_keys, case.new_values, case.token_to_sequence, case.token_positions,
                             case.block_tables, keys, values)
    keys, values = (t[case.block_tables[0].long()].transpose(0, 1).flatten(1, 2).float() for t in (keys, values))
    for row in {*range(10), *range(chunk - 10, chunk)}:
        seen = 66_000 + row + 1
        scores = case.query[row].float().view(kv_heads, -1, 128) @ keys[:, :seen].transpose(1, 2) * case.scale
        want = (scores.softmax(-1) @ values[:, :seen]).reshape(heads, 128)
        assert (out[row].float() - want).abs().max().item() <= ATOL


# 76 to 97 pairs of whole prompts, more than there are clusters of two at once: shared with 19 K/V tiles, and with 12 of each of
# two requests; not with 4 tiles, a table with room for a prefix or a window that ends in the prompt.
@pytest.mark.parametrize("lengths,heads,kv_heads,window,spare", [
    ((2500,), 8, 1, None, 0), ((1540, 1530), 8, 1, None, 0), ((600,) * 4, 8, 1, None, 0), ((2500,), 8, 1, None, 200),
    ((2500,), 8, 1, 700, 0), ((2500,), 8, 1, 2600, 0)], ids=str)
def test_whole_prompts_in_clusters_that_wait(lengths, heads, kv_heads, window, spare, device):
    case = Case(lengths, lengths, heads, kv_heads, 64, 64, window, 16, torch.bfloat16, seed=34)
    case.tables = torch.nn.functional.pad(case.tables, (0, spare), value=-1)
    case.prefill(device)
    case.check()
