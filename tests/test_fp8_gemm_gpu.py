"""FP8 block-scaled linear on the GPU: quantiser bit-exact, GEMM within 1e-2 of the dequantised product.

BASELINE's bound is 1e-2 relative to the dequantised fp32 product for the GEMM
itself (pre-quantised operands); against the CPU restatement of the reference's
kernels the result differs only by fp32 summation order inside a 128-wide block.
"""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import workloads
from mini_inference_engine_b200.engine.kernels import sm89_fp8
from oracle import hot_path

pytestmark = pytest.mark.gpu


def _dequantised_product(a8, a_scale, w8, w_scale):
    """fp64 product of the dequantised operands (benchmarks/commands/run_kernel_track.py:210-217)."""

    m, k = a8.shape
    n = w8.shape[0]
    a = a8.double() * a_scale.double().repeat_interleave(128, dim=1)[:, :k]
    w = w8.double() * w_scale.double().repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)[:, :k]
    return a @ w.T


@pytest.mark.parametrize("m", [1, 5, 130])
@pytest.mark.parametrize("k", [2560, 259, 127])
def test_quantiser_is_bit_exact(m, k, device):
    torch.manual_seed(m * 1000 + k)
    x = torch.randn(m, k).to(torch.bfloat16)
    x[0, ::31] *= 80
    if m > 1:
        x[1] = 0
    if m > 2:
        x[2] *= 1e12
    if m > 3:
        x[3] *= 1e-15
    q_ref, s_ref = hot_path.quantize_activation(x)
    q, s = sm89_fp8.quantize_sm89_fp8_activation(x.to(device))
    assert q.shape == (m, k) and s.shape == (m, (k + 127) // 128)
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))
    assert torch.equal(s.cpu(), s_ref)


@pytest.mark.parametrize("name", ["qkv", "o", "gate_up", "down"])
@pytest.mark.parametrize("m", [1, 8, 64, 256, 2048])
def test_model_shapes_match_dequantised_product(name, m, device, status_clean):
    """BASELINE configuration 1."""

    x, weight = workloads.gemm_case(name, m, seed=0)
    w8, w_scale = hot_path.quantize_weight(weight)
    out = sm89_fp8.sm89_fp8_linear(x.to(device), w8.to(device), w_scale.to(device), block_size=[128, 128])
    torch.cuda.synchronize()
    assert out.shape == (m, w8.shape[0]) and out.dtype == torch.bfloat16
    a8, a_scale = hot_path.quantize_activation(x)
    exact = _dequantised_product(a8, a_scale, w8, w_scale)
    error = (out.cpu().double() - exact).norm(dim=1) / exact.norm(dim=1).clamp_min(1e-30)
    assert error.max().item() < 1e-2, error.max().item()
    if m <= 64:
        port = hot_path.fp8_linear(x, w8, w_scale)
        # Same quantised operands and per-block scaling; only fp32 summation order inside a block differs.
        assert (out.cpu().float() - port.float()).abs().max().item() <= 2e-2 * port.float().abs().max().item()


@pytest.mark.parametrize("m", [1, 3, 17, 100, 128, 129, 255, 300, 1000])
@pytest.mark.parametrize("n,k", [(129, 128), (257, 127), (193, 129), (321, 259), (1024, 2560), (256, 4096)])
def test_tail_shapes_and_row_counts(m, n, k, device, status_clean):
    """N and K tails that cross a scale-block boundary (engine/kernels/sm89_fp8_validation.py:28-31)."""

    generator = torch.Generator().manual_seed(n * 7 + k * 3 + m)
    w8 = (torch.randn(n, k, generator=generator) * 32).clamp(-448, 448).to(torch.float8_e4m3fn)
    w_scale = torch.rand((n + 127) // 128, (k + 127) // 128, generator=generator) * 0.09 + 0.001
    x = torch.randn(m, k, generator=generator)
    x[:, ::31] *= 80
    if m > 1:
        x[1] = 0
    x = x.to(torch.bfloat16)
    out = sm89_fp8.sm89_fp8_linear(x.to(device), w8.to(device), w_scale.to(device), block_size=(128, 128))
    port = hot_path.fp8_linear(x, w8, w_scale)
    scale = port.float().abs().max().item()
    assert (out.cpu().float() - port.float()).abs().max().item() <= 1e-2 * scale
    if m > 1:
        assert not out[1].any()  # an all-zero row stays exactly zero


@pytest.mark.parametrize("m", [65, 81, 128])
@pytest.mark.parametrize("k", [2048, 2064, 2560])
def test_both_numbers_of_promotion_warps(m, k, device, status_clean):
    """Four K blocks a CTA, and five: eight and sixteen warps; token shares of a CTA that the warps do not divide.  Bound: the
    output's rounding to bf16, and fp32 sums of 20 blocks of 128 products."""

    generator = torch.Generator().manual_seed(m + k)
    w8 = (torch.randn(4096, k, generator=generator) * 32).clamp(-448, 448).to(torch.float8_e4m3fn)
    w_scale = torch.rand(32, (k + 127) // 128, generator=generator) * 0.09 + 0.001
    x = torch.randn(m, k, generator=generator).to(torch.bfloat16)
    out = sm89_fp8.sm89_fp8_linear(x.to(device), w8.to(device), w_scale.to(device), block_size=[128, 128])
    exact = _dequantised_product(*hot_path.quantize_activation(x), w8, w_scale)
    error = (out.cpu().double() - exact).abs()
    assert (error <= 2.0 ** -8 * exact.abs() + 2.0 ** -14 * exact.abs().amax()).all()


def test_rows_are_independent_and_bias_dtype(device, status_clean):
    """A row's result does not depend on its neighbours (tests/test_sm89_fp8_exact.py:15-53)."""

    x, weight = workloads.gemm_case("o", 300, seed=3)
    w8, w_scale = hot_path.quantize_weight(weight)
    w8, w_scale, xd = w8.to(device), w_scale.to(device), x.to(device)
    full = sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[128, 128])
    for rows in (1, 7, 130):
        part = sm89_fp8.sm89_fp8_linear(xd[:rows], w8, w_scale, block_size=[128, 128])
        # Small and large row counts take different tile orientations; both apply the same per-block
        # arithmetic, so they agree to fp32 summation order.
        assert (part.float() - full[:rows].float()).abs().max().item() <= 2e-2 * full.float().abs().max().item()
    again = sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[128, 128])
    assert torch.equal(again, full)  # deterministic: stream-K partials are summed in a fixed order
    bias = torch.randn(w8.shape[0], device=device, dtype=torch.bfloat16)
    biased = sm89_fp8.sm89_fp8_linear(xd.half().view(3, 100, -1), w8, w_scale, block_size=[128, 128], bias=bias.half(),
                                      output_dtype=torch.float16)
    assert biased.shape == (3, 100, w8.shape[0]) and biased.dtype == torch.float16
    with pytest.raises(ValueError, match="gemm_config"):
        sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[128, 128], gemm_config=sm89_fp8.SPLIT_GEMM_CONFIGS[0])
    with pytest.raises(ValueError, match="path"):
        sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[128, 128], path="fast")
    with pytest.raises(RuntimeError, match="no fallback"):
        sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[64, 64])


@pytest.mark.parametrize("name", ["qkv", "o", "gate_up", "down"])
def test_rows_do_not_depend_on_the_batch_in_invariant_mode(name, device, status_clean):
    """The reference's row-independence promise (tests/test_sm89_fp8_exact.py): with the K range never cut
    (``set_batch_invariant``), a token's output row is bit-identical whether it is computed alone, in a
    small batch (narrow kernel) or in a large one (wide kernel, partial last round of tiles included)."""

    x, weight = workloads.gemm_case(name, 1000, seed=3)
    w8, w_scale = hot_path.quantize_weight(weight)
    xd, w8, w_scale = x.to(device), w8.to(device), w_scale.to(device)
    previous = sm89_fp8.set_batch_invariant(True)
    try:
        full = sm89_fp8.sm89_fp8_linear(xd, w8, w_scale, block_size=[128, 128])
        for rows in (1, 7, 129):
            part = sm89_fp8.sm89_fp8_linear(xd[:rows], w8, w_scale, block_size=[128, 128])
            assert torch.equal(part, full[:rows]), (name, rows)
        single = sm89_fp8.sm89_fp8_linear(xd[999:1000], w8, w_scale, block_size=[128, 128])
        assert torch.equal(single, full[999:1000])
    finally:
        sm89_fp8.set_batch_invariant(previous)


@pytest.mark.parametrize("m", [1, 40, 300])
def test_weights_written_by_queued_kernels_are_read_after_them(m, device, status_clean):
    """A product without the static-weights promise reads weights that a kernel two launches ahead of it writes."""

    from mini_inference_engine_b200 import _lib
    from mini_inference_engine_b200.engine.kernels.decoder_glue import softcap_

    n, k = 19456, 2560
    lib, stream = _lib.load(), _lib.stream_arg(device)
    generator = torch.Generator(device=device).manual_seed(m)
    sources = [torch.randn(n, k, generator=generator, device=device).to(torch.bfloat16) for _ in range(2)]
    q, scales = sm89_fp8.quantize_activation_kmajor(torch.randn(m, k, generator=generator, device=device).bfloat16())
    w8, row_scales = torch.empty(n, k, dtype=torch.float8_e4m3fn, device=device), torch.empty(k // 128, n, device=device)
    w_scale, between = torch.full((n // 128, k // 128), 1e-3, device=device), torch.ones(4, device=device)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=device)

    def step(source, wait):
        _lib.check(lib.mie_fp8_quantize(_lib.ptr(source), k, _lib.DTYPE_CODES[source.dtype], _lib.ptr(w8), k,
                                        _lib.ptr(row_scales), n, n, k, stream))
        softcap_(between, 30.0)
        if wait:
            torch.cuda.synchronize()
        sm89_fp8.launch_fp8_gemm(q, scales, w8, w_scale, out, m, k)
        return out.clone()

    want = [step(source, True) for source in sources]
    assert not torch.equal(*want)
    for i in range(40):
        assert torch.equal(step(sources[i % 2], False), want[i % 2])
