"""Projections that finish their own rows: equal to the projection followed by the row kernel."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import _lib
from mini_inference_engine_b200.engine.kernels import sm89_fp8

pytestmark = pytest.mark.gpu


def _operands(m, n, k, device):
    generator = torch.Generator(device=device).manual_seed(n + k + m)
    w8 = (torch.randn(n, k, generator=generator, device=device) * 32).clamp(-448, 448).to(torch.float8_e4m3fn)
    w_scale = torch.rand(n // 128, -(-k // 128), generator=generator, device=device) * 2e-3 + 1e-4
    x = torch.randn(m, k, generator=generator, device=device).to(torch.bfloat16)
    x[0] *= 0.0 if m > 1 else 1.0
    q, scales = sm89_fp8.quantize_activation_kmajor(x)
    return q, scales, w8, w_scale


def _product(q, scales, w8, w_scale, m, k, max_split):
    out = torch.empty(m, w8.shape[0], dtype=torch.bfloat16, device=q.device)
    sm89_fp8.launch_fp8_gemm(q, scales, w8, w_scale, out, m, k, max_split=max_split)
    return out


# Tokens at the edges of the column tiles; a K that is cut in parts, one of a single block, one with a tail.
SIZES = [(m, k) for m in (1, 15, 16, 17, 32, 33, 64, 65, 128) for k in (128, 1024, 2560)] + [(5, 2032), (40, 9728)]


@pytest.mark.parametrize("m,k", SIZES)
@pytest.mark.parametrize("max_split", [0, 1])
def test_gated_rows(m, k, max_split, device, status_clean):
    cols = 384
    q, scales, w8, w_scale = _operands(m, 2 * cols, k, device)
    lib, stream = _lib.load(), _lib.stream_arg(device)
    assert lib.mie_fp8_gemm_finishes(m, 2 * cols)
    got, got_s = torch.zeros(m, cols, dtype=torch.uint8, device=device), torch.zeros(3, m + 2, device=device)
    _lib.check(lib.mie_fp8_gemm_silu(
        _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), k, _lib.ptr(w_scale), w_scale.stride(0),
        _lib.ptr(got), cols, _lib.ptr(got_s), m + 2, m, cols, k, max_split, 0, _lib.ptr(_lib.status_word(device)), stream))
    both = _product(q, scales, w8, w_scale, m, k, max_split)
    want, want_s = torch.zeros_like(got), torch.zeros_like(got_s)
    _lib.check(lib.mie_silu_mul(_lib.ptr(both), _lib.ptr(both[:, cols:]), 2 * cols, None, _lib.ptr(want), cols,
                                _lib.ptr(want_s), m + 2, m, cols, stream))
    torch.cuda.synchronize()
    if max_split == 1:  # the same sums in the same order
        assert torch.equal(got, want) and torch.equal(got_s, want_s)
        return
    # K may be cut elsewhere: fp32 sums in another order, which can move a bf16 rounding (2^-8) and through it an e4m3
    # one (2^-3 of a value, at most one step).
    full = got.view(torch.float8_e4m3fn).float() * got_s[:, :m].t().repeat_interleave(128, 1)
    ref = want.view(torch.float8_e4m3fn).float() * want_s[:, :m].t().repeat_interleave(128, 1)
    top = want_s[:, :m].t().repeat_interleave(128, 1) * 448
    assert ((full - ref).abs() <= 0.13 * ref.abs() + 2 ** -8 * top).all()
    assert ((full - ref).norm() <= 1e-2 * ref.norm()).all()


@pytest.mark.parametrize("m,k", SIZES)
@pytest.mark.parametrize("heads", [(4, 2), (3, 1)])
@pytest.mark.parametrize("kv8", [False, True])
def test_cache_rows(m, k, heads, kv8, device, status_clean):
    from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3Shape, rope_table

    q_heads, kv_heads = heads
    n, pages, width = (q_heads + 2 * kv_heads) * 128, m + 3, 2
    q, scales, w8, w_scale = _operands(m, n, k, device)
    lib, stream, status = _lib.load(), _lib.stream_arg(device), _lib.status_word(device)
    norms = [(1 + 0.1 * torch.randn(128, device=device)).to(torch.bfloat16) for _ in range(2)]
    rope = rope_table(Qwen3Shape(), 64, device)
    positions = torch.arange(m, dtype=torch.int32, device=device) % 32
    tables = torch.randperm(pages, device=device)[:m].to(torch.int32)[:, None].repeat(1, width).contiguous()
    meta = (_lib.ptr(norms[0]), _lib.ptr(norms[1]), _lib.ptr(rope), 64, _lib.index_arg(positions), _lib.index_arg(None),
            _lib.index_arg(tables))
    results = []
    for fused in (True, False):
        queries = torch.zeros(m, q_heads, 128, dtype=torch.bfloat16, device=device)
        keys = torch.zeros(pages, kv_heads, 16, 128, dtype=torch.bfloat16, device=device)
        values, pool = torch.zeros_like(keys), torch.zeros(pages, kv_heads, 2, 16, 128, dtype=torch.uint8, device=device)
        pool_s = torch.zeros(pages, kv_heads, 2, 16, device=device)
        views = (_lib.view4_arg(keys), _lib.view4_arg(values))
        if fused:
            _lib.check(lib.mie_fp8_gemm_qkv(
                _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), k, _lib.ptr(w_scale),
                w_scale.stride(0), *meta, _lib.ptr(queries), *views, _lib.ptr(pool) if kv8 else None, kv_heads * 4096,
                _lib.ptr(pool_s), m, k, q_heads, kv_heads, 16, pages, m, width, 1e-6, 1, 0, _lib.ptr(status), stream))
        else:
            rows = _product(q, scales, w8, w_scale, m, k, 1)
            tail = (m, q_heads, kv_heads)
            if kv8:
                _lib.check(lib.mie_qkv_norm_rope_write_kv8(_lib.ptr(rows), n, *meta, _lib.ptr(queries), _lib.ptr(pool),
                                                           kv_heads * 4096, _lib.ptr(pool_s), *tail, pages, m, width, 1e-6,
                                                           _lib.ptr(status), stream))
            else:
                _lib.check(lib.mie_qkv_norm_rope_write(_lib.ptr(rows), n, *meta, _lib.ptr(queries), *views, *tail, 16,
                                                       pages, m, width, 1e-6, _lib.ptr(status), stream))
        results.append((queries, keys, values, pool, pool_s))
    torch.cuda.synchronize()
    # The projected rows are the same, and so is every sum and rounding after them.
    for got, want in zip(*results):
        assert torch.equal(got, want)


def test_cached_rows_do_not_depend_on_the_step_they_come_in(device, status_clean):
    """The same projected rows in a step that finishes them in the projection and in one that does not: a sum of squares
    added in another order would move a bf16 rounding of some of these two million entries."""

    m, k, q_heads, kv_heads = 128, 128, 32, 8
    n = (q_heads + 2 * kv_heads) * 128
    from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3Shape, rope_table

    lib, stream, status = _lib.load(), _lib.stream_arg(device), _lib.status_word(device)
    rope, norm = rope_table(Qwen3Shape(), 64, device), torch.ones(128, dtype=torch.bfloat16, device=device)
    positions, tables = torch.zeros(m, dtype=torch.int32, device=device), torch.arange(m, dtype=torch.int32, device=device)[:, None]
    meta = (_lib.ptr(norm), _lib.ptr(norm), _lib.ptr(rope), 64, _lib.index_arg(positions), _lib.index_arg(None),
            _lib.index_arg(tables))
    for seed in range(3):
        torch.manual_seed(seed)
        q, scales, w8, w_scale = _operands(m, n, k, device)
        w_scale.copy_(torch.rand_like(w_scale) * 1e-2)
        rows = _product(q, scales, w8, w_scale, m, k, 1)
        out = [torch.zeros(m, q_heads, 128, dtype=torch.bfloat16, device=device) for _ in range(2)]
        keys = [torch.zeros(m, kv_heads, 16, 128, dtype=torch.bfloat16, device=device) for _ in range(2)]
        values = torch.zeros_like(keys[0])
        _lib.check(lib.mie_fp8_gemm_qkv(
            _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), k, _lib.ptr(w_scale),
            w_scale.stride(0), *meta, _lib.ptr(out[0]), _lib.view4_arg(keys[0]), _lib.view4_arg(values), None, 0, None, m, k,
            q_heads, kv_heads, 16, m, m, 1, 1e-6, 1, 0, _lib.ptr(status), stream))
        _lib.check(lib.mie_qkv_norm_rope_write(_lib.ptr(rows), n, *meta, _lib.ptr(out[1]), _lib.view4_arg(keys[1]),
                                               _lib.view4_arg(values), m, q_heads, kv_heads, 16, m, m, 1, 1e-6,
                                               _lib.ptr(status), stream))
        assert torch.equal(out[0], out[1]) and torch.equal(keys[0], keys[1])


def test_sizes_that_are_not_finished_are_refused(device):
    q, scales, w8, w_scale = _operands(130, 768, 256, device)
    out, out_s = torch.zeros(130, 384, dtype=torch.uint8, device=device), torch.zeros(3, 130, device=device)
    lib = _lib.load()
    assert not lib.mie_fp8_gemm_finishes(130, 768) and not lib.mie_fp8_gemm_finishes(33, 128 * 400)
    with pytest.raises(Exception, match="not finished in the projection"):
        _lib.check(lib.mie_fp8_gemm_silu(
            _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), 256, _lib.ptr(w_scale), 2,
            _lib.ptr(out), 384, _lib.ptr(out_s), 130, 130, 384, 256, 0, 0, _lib.ptr(_lib.status_word(device)),
            _lib.stream_arg(device)))


@pytest.mark.parametrize("m,n,k", [(1, 2560, 9728), (24, 2560, 9728), (300, 1024, 2560)])
def test_repeated_products_are_identical(m, n, k, device, status_clean):
    """Two threads issue alternate K blocks over an odd number of stages: none may take a stage before its block landed,
    however late the operands come (L2 is flushed in between)."""

    q, scales, w8, w_scale = _operands(m, n, k, device)
    first = _product(q, scales, w8, w_scale, m, k, 0)
    flush = torch.empty(160 << 20, dtype=torch.uint8, device=device)
    different = torch.zeros((), dtype=torch.int64, device=device)
    for _ in range(200):
        flush.zero_()
        different += (_product(q, scales, w8, w_scale, m, k, 0) != first).any()
    assert int(different.item()) == 0


# Token tiles that are whole, ragged and single; more tiles than SMs; K of one block, two, and one with a tail.
WIDE = [(m, cols, k) for m in (1, 128, 129, 300) for cols, k in ((128, 128), (384, 256), (640, 2032))] + [(1000, 2560, 384)]


@pytest.mark.parametrize("m,cols,k", WIDE)
def test_gated_rows_of_long_steps(m, cols, k, device, status_clean):
    """The same sums in the same order as the product that is not cut, and the same rounding points: equal bits."""

    q, scales, w8, w_scale = _operands(m, 2 * cols, k, device)
    lib, stream, groups = _lib.load(), _lib.stream_arg(device), cols // 128
    got, got_s = torch.zeros(m, cols, dtype=torch.uint8, device=device), torch.zeros(groups, m + 2, device=device)
    for _ in range(3):
        _lib.check(lib.mie_fp8_gemm_silu_wide(
            _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), w8.stride(0), _lib.ptr(w_scale),
            w_scale.stride(0), _lib.ptr(got), cols, _lib.ptr(got_s), m + 2, m, cols, k, 0,
            _lib.ptr(_lib.status_word(device)), stream))
    both = _product(q, scales, w8, w_scale, m, k, 1)
    want, want_s = torch.zeros_like(got), torch.zeros_like(got_s)
    _lib.check(lib.mie_silu_mul(_lib.ptr(both), _lib.ptr(both[:, cols:]), 2 * cols, None, _lib.ptr(want), cols,
                                _lib.ptr(want_s), m + 2, m, cols, stream))
    assert torch.equal(got, want) and torch.equal(got_s, want_s)


# Tokens, columns, K; whether the wide kernel finishes them, on a GPU of 148 SMs: no cut tail, many rounds; one round, two,
# and three or more of longer sums in front of a cut tail; narrow steps; columns of no whole group.
WIDE_RULE = [(300, 9728, 2560, 1), (12032, 9728, 2560, 1), (200, 9728, 2560, 0), (400, 9728, 2560, 1), (768, 9728, 3072, 0),
             (1536, 9728, 3072, 1), (1024, 9728, 4096, 0), (2048, 9728, 4096, 1), (64, 9216, 2560, 0), (300, 9729, 2560, 0)]


@pytest.mark.parametrize("m,cols,k,pays", WIDE_RULE)
def test_rule_for_gated_rows_of_long_steps(m, cols, k, pays, device):
    lib = _lib.load()
    if int(lib.mie_sm_count()) != 148:
        pytest.skip("measured on 148 SMs")
    assert int(lib.mie_fp8_gemm_silu_wide_pays(m, cols, k, 0)) == pays
