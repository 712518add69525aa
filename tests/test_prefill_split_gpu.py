"""Prefill attention where a cluster shares a pair of query tiles (its K/V tiles, or one query tile each)."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import _lib, workloads
from test_prefill_attention_gpu import ATOL, _oracle, _run
from test_sink_attention_gpu import Case

pytestmark = pytest.mark.gpu

# prefixes, chunks, query and key/value heads: six and eight ranks for one query tile; two ranks beside a request with too
# few tiles; the first tile count that is shared (eight) and the last that is not; a rank per query tile; query tiles that
# end in different K/V tiles; groups of 1, 2 and 8 heads.
SHARED = [
    ((3000,), (16,), 32, 8), ((4100,), (1,), 8, 2), ((1673, 375), (386, 126), 32, 8), ((992, 960), (32, 64), 8, 2),
    ((500, 0), (100, 97), 32, 8), ((1500,), (300,), 8, 8), ((2040,), (129,), 4, 2), ((900, 1500), (33, 200), 8, 1),
]


@pytest.mark.parametrize("shape", SHARED, ids=str)
def test_ranks_of_a_pair(shape, device, status_clean):
    """Bound as for the unshared kernel: bf16 probabilities and outputs of unit values."""

    prefixes, chunks, heads, kv_heads = shape
    case = workloads.prefill_case(seed=11, prefix_lengths=prefixes, chunk_lengths=chunks, q_heads=heads,
                                  kv_heads=kv_heads)
    _, _, expected = _oracle(case)
    _, out = _run(case, device)
    assert (out.float() - expected.float()).abs().max().item() <= ATOL


# length and new tokens of each request; heads, key/value heads, dim, vdim, window; sinks.
WIDE = [
    ([(2500, 40), (1200, 130)], (8, 2, 128, 128, None), "random"), ([(2500, 40)], (4, 4, 192, 128, None), "large"),
    ([(2600, 90)], (8, 2, 128, 128, 1024), "none"), ([(1400, 300)], (4, 2, 64, 64, 1100), "random"),
    ([(1500, 20)], (2, 1, 72, 200, None), "zeros"), ([(1300, 260)], (3, 3, 256, 256, 1030), "random"),
]


@pytest.mark.parametrize("spans,sizes,sinks", WIDE, ids=str)
def test_ranks_with_sinks_and_windows(spans, sizes, sinks, device):
    """Only the first rank counts the sink; a rank may see no key of a windowed row."""

    case = Case([n for n, _ in spans], [c for _, c in spans], *sizes, 16, torch.bfloat16, seed=12, sinks=sinks)
    case.prefill(device)
    case.check()


# Groups of one and four heads, five to eight ranks; with NaN queries a rank has nothing but -inf as its maximum.
@pytest.mark.parametrize("sizes", [(4, 4, 128, 128), (8, 2, 64, 64)], ids=str)
def test_what_is_no_number_reaches_the_result(sizes, device):
    """As without a split: a NaN query gives a NaN row, an infinite value no finite number, whatever its weight."""

    case = Case([2600], [24], *sizes, None, 16, torch.bfloat16, seed=13, sinks="none")
    case.queries[0][5] = float("nan")
    page, slot = int(case.tables[0, 3]), 7  # a token of the first rank, and one that all but a few ranks lie behind
    case.values[page, :, slot, 10] = float("inf")
    case.keys[page, :, slot] *= 0.0
    case.prefill(device)
    bad = ~torch.isfinite(case.out.cpu().float())
    want = torch.zeros_like(bad)
    want[5] = True
    want[..., 10] = True
    assert torch.equal(bad, want) and bool(case.out[5].isnan().all())


@pytest.mark.parametrize("total", [None, 0, 530])
def test_ragged_chunks_with_and_without_their_number_of_tokens(total, device):
    """One long chunk among short ones: by the older entry point, and by the packed one that may know the tokens."""

    case = Case([2500, 40, 700], [500, 20, 10], 8, 4, 128, 128, None, 16, torch.bfloat16, seed=14)
    keys, values, tables = case.on(device)
    cu = torch.tensor([0, 500, 520, 530], dtype=torch.int32, device=device)
    lens = torch.tensor(case.lengths, dtype=torch.int32, device=device)
    lib, name = _lib.load(), "mie_sink_prefill_attention" if total is None else "mie_sink_prefill_packed"
    _lib.check(getattr(lib, name)(
        _lib.ptr(case.q), case.q.stride(0), case.q.stride(1), _lib.ptr(case.out), case.out.stride(0), case.out.stride(1),
        _lib.view4_arg(keys), _lib.view4_arg(values), _lib.index_arg(tables), _lib.index_arg(cu), _lib.index_arg(lens),
        *(() if total is None else (total,)), 3, 500, 8, 4, 128, 128, 16, case.pages, int(tables.shape[1]),
        _lib.DTYPE_CODES[torch.bfloat16], case.scale, 0, _lib.ptr(case.common["sinks"]), _lib.ptr(case.status),
        _lib.stream_arg(device)))
    case.check()


@pytest.mark.parametrize("heads,kv_heads,others", [(32, 8, 11), (8, 8, 11)])
def test_alone_and_among_many(heads, kv_heads, others, device, status_clean):
    """Alone a chunk is shared by six ranks, among eleven like it (96 pairs) by none: both within the bound, and their sums
    in another order, which some of their bits show."""

    sizes = dict(q_heads=heads, kv_heads=kv_heads)
    alone = workloads.prefill_case(seed=15, prefix_lengths=(3000,), chunk_lengths=(16,), **sizes)
    many = workloads.prefill_case(seed=15, prefix_lengths=(3000,) * (others + 1), chunk_lengths=(16,) * (others + 1), **sizes)
    many.query[:16] = alone.query
    many.new_keys[:, :, :16], many.new_values[:, :, :16] = alone.new_keys, alone.new_values
    _, _, expected = _oracle(alone)
    results = [_run(case, device)[1][:16].float() for case in (alone, many)]
    for out in results:
        assert (out - expected.float()).abs().max().item() <= ATOL
    assert not torch.equal(*results)
