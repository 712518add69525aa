"""Prefill attention where a CTA has a pair of query tiles to itself: steps with pairs enough for the GPU."""

from __future__ import annotations

import pytest
import torch

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
