"""Decode attention of few requests, each KV head of a request shared by a cluster."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import _lib, workloads
from mini_inference_engine_b200.engine.kv_cache import triton_paged_decode_attention
from mini_inference_engine_b200.engine.kv_cache.triton_paged_attention import decode_scratch, launch_decode_attention
from oracle import hot_path
from test_sink_attention_gpu import Case

pytestmark = pytest.mark.gpu

# Lengths and heads: eight, four, two and one CTA a head; fewer tiles than warps; one tile; groups of 1, 3 and 8 heads.
BATCHES = [((611,), 32, 8), ((1,), 32, 8), ((129, 16, 3000), 32, 8), ((17, 65, 1000, 300, 80, 31), 16, 8),
           ((900, 33, 15, 16, 640, 128, 127, 2, 1, 700, 64, 90), 8, 8), ((2100,), 8, 1), ((333, 1), 24, 8)]


@pytest.mark.parametrize("lengths,heads,kv_heads", BATCHES, ids=str)
def test_shared_requests(lengths, heads, kv_heads, device, status_clean):
    """Bound of the queue's path: bf16 outputs of unit values."""

    case = workloads.decode_case(lengths, seed=21, q_heads=heads, kv_heads=kv_heads)
    dev = case.to(device)
    out = triton_paged_decode_attention(dev.query, dev.key_blocks, dev.value_blocks, dev.block_tables,
                                        dev.sequence_lengths, scale=case.scale)
    expected = hot_path.paged_decode_attention(case.query, case.key_blocks, case.value_blocks, case.block_tables,
                                               case.sequence_lengths, case.scale)
    assert (out.cpu().float() - expected.float()).abs().max().item() <= 2e-2


# heads, kv_heads, dim, vdim, window; sinks.
WIDE = [((8, 2, 128, 128, None), "large"), ((20, 1, 16, 64, 129), "random"), ((4, 4, 256, 256, 50), "zeros"),
        ((5, 1, 72, 200, 1), "none"), ((6, 2, 40, 24, 16), "random")]


@pytest.mark.parametrize("sizes,sinks", WIDE, ids=str)
def test_shared_sinks_and_windows(sizes, sinks, device):
    case = Case([700, 1, 16, 130], [1] * 4, *sizes, 16, torch.bfloat16, seed=22, sinks=sinks)
    case.decode(device)
    case.check()


def _launches(call) -> int:
    lib = _lib.load()
    before = int(lib.mie_launch_count())
    call()
    return int(lib.mie_launch_count()) - before


# As above without the table that has room for one chunk only, which is not shared; one token in a wide table instead.
SHARED = [*(b for b in BATCHES if b[0] != (1,)), ((1,), 32, 8)]


@pytest.mark.parametrize("lengths,heads,kv_heads", SHARED, ids=str)
def test_one_launch_and_no_plan(lengths, heads, kv_heads, device, status_clean):
    """A shared call is one launch; calls that reuse its plan get the result, whichever way they take."""

    case = workloads.decode_case(lengths, seed=23, q_heads=heads, kv_heads=kv_heads)
    dev = case.to(device)
    tables = torch.nn.functional.pad(dev.block_tables, (0, 6), value=-1)
    out = torch.empty_like(dev.query)
    scratch = decode_scratch(len(lengths), heads, kv_heads, 128, sum(lengths), device)
    scratch.fill_(0x5A)

    def attend(**how):
        out.fill_(float("nan"))
        launch_decode_attention(dev.query, out, dev.key_blocks, dev.value_blocks, tables, dev.sequence_lengths, None,
                                scale=case.scale, max_total_tokens=sum(lengths), scratch=scratch, **how)
        return out.cpu().float().transpose(1, 2)  # as the operator returns it

    expected = hot_path.paged_decode_attention(case.query, case.key_blocks, case.value_blocks, case.block_tables,
                                               case.sequence_lengths, case.scale).float()
    results = []
    assert _launches(lambda: results.append(attend(split_policy=1))) == 1
    assert _launches(lambda: results.append(attend(split_policy=1, use_plan=True, plan_slot=1))) == 1
    results.append(attend(split_policy=0, use_plan=True, plan_slot=2))  # not shared
    assert _launches(lambda: results.append(attend(split_policy=64))) >= 3
    for result in results:
        assert (result - expected).abs().max().item() <= 2e-2


@pytest.mark.parametrize("sizes,sinks", WIDE, ids=str)
def test_one_launch_with_sinks_and_windows(sizes, sinks, device):
    """Windows of up to 48 tokens are one chunk a request, which a warp takes: plan, queue and merge."""

    case = Case([700, 1, 16, 130], [1] * 4, *sizes, 16, torch.bfloat16, seed=24, sinks=sinks)
    calls = _launches(lambda: case.decode(device))  # one call, and one that reuses its plan
    assert calls == (2 if sizes[4] is None or sizes[4] > 48 else 3 + 2)
    case.check()
