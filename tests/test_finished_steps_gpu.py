"""Whole steps whose projections finish their own rows, as real models' do: the tests of the small models, whose weights
otherwise keep the separate launches, once more with every product that can finishing its rows."""

from __future__ import annotations

import pytest
import torch

import test_continuous_gpu
import test_decode_step_gpu
import test_fp8_kv_gpu
from mini_inference_engine_b200 import _lib
from mini_inference_engine_b200.engine.kernels import sm89_fp8
from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3DecodeRunner, Qwen3Weights

pytestmark = pytest.mark.gpu


@pytest.fixture()
def finished(monkeypatch):
    """Rows are finished wherever that is possible; afterwards both kinds must have been, equally often."""

    taken = {"mie_fp8_gemm_silu": 0, "mie_fp8_gemm_qkv": 0}
    lib = _lib.load()
    monkeypatch.setattr(sm89_fp8, "finishes_rows",
                        lambda weight, m, *, gated: bool(lib.mie_fp8_gemm_finishes(m, int(weight.shape[0]))))
    for name in taken:
        def counting(*args, _name=name, _call=getattr(lib, name)):
            taken[_name] += 1
            return _call(*args)

        monkeypatch.setattr(lib, name, counting)
    yield taken
    assert taken["mie_fp8_gemm_silu"] == taken["mie_fp8_gemm_qkv"] > 0


@pytest.mark.parametrize("use_graph", [False, True])
def test_decode_steps(use_graph, device, finished):
    test_decode_step_gpu.test_tokens_within_the_noise_band_on_random_state(use_graph, device)


def test_generation(device, finished):
    test_decode_step_gpu.test_generation_tokens_equal_the_oracle(device)


@pytest.mark.parametrize("use_graphs", [True, False])
def test_continuous_batching(use_graphs, device, finished):
    test_continuous_gpu.test_requests_finish_at_different_times_through_shrinking_buckets(use_graphs, device)


@pytest.mark.parametrize("use_graphs", [True, False])
def test_mixed_steps(use_graphs, device, finished):
    test_continuous_gpu.test_prompt_chunks_ride_along_with_decode_rows(use_graphs, device)


def test_bucket_graphs(device, finished):
    test_continuous_gpu.test_bucket_graph_equals_the_eager_step_bit_for_bit(device)


@pytest.mark.parametrize("mixed", [False, True])
def test_shared_prefix_pages(mixed, device, finished):
    test_continuous_gpu.test_requests_sharing_prefix_pages_run_through_the_captured_steps(mixed, device)


def test_decode_over_the_fp8_cache(device, finished):
    test_fp8_kv_gpu.test_decode_step_over_the_fp8_cache(device)


def test_prompt_chunks_over_the_fp8_cache(device, finished):
    test_fp8_kv_gpu.test_prompt_chunks_over_the_fp8_cache(device)


@pytest.mark.parametrize("mixed", [False, True])
def test_generation_over_the_fp8_cache(mixed, device, finished):
    test_fp8_kv_gpu.test_generation_over_the_fp8_cache_equals_the_oracle(mixed, device)


def test_launch_count(device, finished):
    """Two launches a layer fewer than with separate row kernels: q/k/v rows and SiLU * up are part of their products."""

    shape = test_decode_step_gpu.SHAPE
    runner = Qwen3DecodeRunner(Qwen3Weights(shape, device, seed=1), num_pages=8, max_batch=1, max_context=64)
    runner.decode_forward(torch.tensor([1], device=device), torch.tensor([3], dtype=torch.int32, device=device),
                          torch.arange(4, dtype=torch.int32, device=device).view(1, 4))
    assert runner.launches_per_step == shape.layers * 8 + 2 + 2


@pytest.mark.parametrize("kv8", [False, True])
def test_rows_of_any_owner_position_and_page(kv8, device):
    """Owners of a mixed step, and metadata that the step does not allow: the finished projection writes the pages and
    sets the status bits that the projection and the row kernel do."""

    from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3Shape, rope_table

    m, k, q_heads, kv_heads, pages = 9, 256, 2, 1, 6
    n = (q_heads + 2 * kv_heads) * 128
    generator = torch.Generator(device=device).manual_seed(3)
    w8 = (torch.randn(n, k, generator=generator, device=device) * 32).clamp(-448, 448).to(torch.float8_e4m3fn)
    w_scale = torch.rand(n // 128, k // 128, generator=generator, device=device) * 2e-3 + 1e-4
    q, scales = sm89_fp8.quantize_activation_kmajor(torch.randn(m, k, generator=generator, device=device).bfloat16())
    rows = torch.empty(m, n, dtype=torch.bfloat16, device=device)
    sm89_fp8.launch_fp8_gemm(q, scales, w8, w_scale, rows, m, k, max_split=1)
    norm, rope = torch.ones(128, dtype=torch.bfloat16, device=device), rope_table(Qwen3Shape(), 64, device)
    lib, stream = _lib.load(), _lib.stream_arg(device)
    good = dict(owner=[0, 1, 2, 2, 2, 0, 1, 1, 2], position=[3, 0, 16, 17, 31, 4, 1, 2, 15],
                table=[[5, -1], [2, -1], [0, 4]])
    bad = {
        0: {}, _lib.STATUS_BAD_POSITION: {"position": [3, -1, 16, 17, 70, 4, 1, 33, 15]},
        _lib.STATUS_BAD_SEQUENCE: {"owner": [0, 1, 2, 3, 2, -1, 1, 1, 2]},
        _lib.STATUS_BAD_PAGE: {"table": [[5, -1], [2, -1], [6, -3]]},
    }
    for bits, change in bad.items():
        meta = {**good, **change}
        owner, position, table = (torch.tensor(meta[name], dtype=torch.int32, device=device)
                                  for name in ("owner", "position", "table"))
        shared = (_lib.ptr(norm), _lib.ptr(norm), _lib.ptr(rope), 64, _lib.index_arg(position), _lib.index_arg(owner),
                  _lib.index_arg(table))
        results = []
        for fused in (True, False):
            status = torch.zeros(1, dtype=torch.int32, device=device)
            queries = torch.zeros(m, q_heads, 128, dtype=torch.bfloat16, device=device)
            keys = torch.zeros(pages, kv_heads, 16, 128, dtype=torch.bfloat16, device=device)
            values, pool = torch.zeros_like(keys), torch.zeros(pages, kv_heads, 2, 16, 128, dtype=torch.uint8, device=device)
            pool_s = torch.zeros(pages, kv_heads, 2, 16, device=device)
            views = (_lib.view4_arg(keys), _lib.view4_arg(values))
            if fused:
                _lib.check(lib.mie_fp8_gemm_qkv(
                    _lib.ptr(q), q.stride(0), _lib.ptr(scales), scales.stride(0), _lib.ptr(w8), k, _lib.ptr(w_scale),
                    w_scale.stride(0), *shared, _lib.ptr(queries), *views, _lib.ptr(pool) if kv8 else None,
                    kv_heads * 4096, _lib.ptr(pool_s), m, k, q_heads, kv_heads, 16, pages, 3, 2, 1e-6, 1, 0,
                    _lib.ptr(status), stream))
            elif kv8:
                _lib.check(lib.mie_qkv_norm_rope_write_kv8(
                    _lib.ptr(rows), n, *shared, _lib.ptr(queries), _lib.ptr(pool), kv_heads * 4096, _lib.ptr(pool_s), m,
                    q_heads, kv_heads, pages, 3, 2, 1e-6, _lib.ptr(status), stream))
            else:
                _lib.check(lib.mie_qkv_norm_rope_write(
                    _lib.ptr(rows), n, *shared, _lib.ptr(queries), *views, m, q_heads, kv_heads, 16, pages, 3, 2, 1e-6,
                    _lib.ptr(status), stream))
            results.append((queries, keys, values, pool, pool_s, status))
        for got, want in zip(*results):
            assert torch.equal(got, want)
        assert int(results[0][-1].item()) == bits
        written = results[0][3] if kv8 else results[0][1]
        assert bool(written.any())
