"""Row kernels at the sizes where their lanes, alignments and quotients can go wrong."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200 import _lib
from mini_inference_engine_b200.engine.kernels import sm89_fp8
from oracle import hot_path

pytestmark = pytest.mark.gpu


def test_quotients_of_the_quantiser_are_ieee_quotients(device):
    """Zeros of both signs, tiny and huge groups, infinities and NaN: the bytes of an IEEE division."""

    torch.manual_seed(0)
    x = torch.randn(64, 256).to(torch.bfloat16)
    x[0], x[1], x[2, ::2], x[3] = 0.0, -0.0, -0.0, x[3] * 1e-37
    x[4] *= 3e37
    x[5, 7], x[6, 9], x[7, 11] = float("inf"), float("-inf"), float("nan")
    x[8:24] *= torch.exp(torch.linspace(-30, 30, 16))[:, None].to(torch.bfloat16)
    got, scales = sm89_fp8.quantize_sm89_fp8_activation(x.to(device))
    groups = x.float().view(64, 2, 128)
    want_scale = torch.nan_to_num(groups.abs(), nan=0.0, posinf=float("inf")).amax(-1) / 448.0
    want = (groups / want_scale.clamp_min(1e-12)[..., None]).view(64, 256)
    # the conversion saturates where torch's overflows to NaN; both keep NaN
    want = torch.where(want.isnan(), want, want.clamp(-448, 448)).to(torch.float8_e4m3fn)
    assert torch.equal(scales.cpu(), want_scale)
    nan = want.float().isnan()
    assert torch.equal(got.cpu().float().isnan(), nan)
    assert torch.equal(got.cpu().view(torch.uint8)[~nan], want.view(torch.uint8)[~nan])


@pytest.mark.parametrize("heads", [(1, 1), (3, 1), (16, 8), (32, 8), (40, 20)])
@pytest.mark.parametrize("offset", [0, 4])  # rows aligned to 16 bytes, and to 8 only
def test_qkv_rows_of_odd_head_counts_and_alignments(heads, offset, device, status_clean):
    """Half-warps of different head kinds share a warp; the e4m3 pool holds the quantised bf16 rows."""

    from mini_inference_engine_b200.engine.model_runner.qwen3_decode import Qwen3Shape, rope_table

    torch.manual_seed(1)
    q_heads, kv_heads = heads
    tokens, pages, width = 5, 4, (q_heads + 2 * kv_heads) * 128
    rows = torch.randn(tokens, width + 8).to(torch.bfloat16)
    qkv = rows[:, offset:offset + width]
    weights = [(1 + 0.1 * torch.randn(128)).to(torch.bfloat16) for _ in range(2)]
    positions = torch.tensor([0, 17, 18, 31, 40], dtype=torch.int32)
    owners = torch.zeros(tokens, dtype=torch.int32)
    tables = torch.tensor([[2, 0, 3]], dtype=torch.int32)
    q, k, v = (part.reshape(1, tokens, -1, 128) for part in qkv.split([q_heads * 128, kv_heads * 128, kv_heads * 128], 1))
    cos, sin = hot_path.rope_cos_sin(positions.view(1, tokens), 128, 5_000_000.0)
    q_want, k_want = hot_path.apply_rotary_pos_emb(hot_path.rms_norm(q, weights[0], 1e-6).transpose(1, 2),
                                                   hot_path.rms_norm(k, weights[1], 1e-6).transpose(1, 2), cos, sin)
    keys_want = torch.zeros(pages, kv_heads, 16, 128, dtype=torch.bfloat16)
    values_want = torch.zeros_like(keys_want)
    hot_path.write_packed_kv(k_want, v.transpose(1, 2), owners, positions, tables, keys_want, values_want)

    d_rows = rows.to(device)
    d_qkv, d_w = d_rows[:, offset:offset + width], [w.to(device) for w in weights]
    rope, status = rope_table(Qwen3Shape(), 64, device), _lib.status_word(device)
    keys = torch.zeros(pages, kv_heads, 16, 128, dtype=torch.bfloat16, device=device)
    values, queries = torch.zeros_like(keys), torch.empty(tokens, q_heads, 128, dtype=torch.bfloat16, device=device)
    meta = [t.to(device) for t in (positions, owners, tables)]
    common = (_lib.ptr(d_qkv), d_qkv.stride(0), _lib.ptr(d_w[0]), _lib.ptr(d_w[1]), _lib.ptr(rope), 64,
              *(_lib.index_arg(t) for t in meta), _lib.ptr(queries))
    tail = (tokens, q_heads, kv_heads)
    _lib.check(_lib.load().mie_qkv_norm_rope_write(*common, _lib.view4_arg(keys), _lib.view4_arg(values), *tail, 16, pages,
                                                   1, 3, 1e-6, _lib.ptr(status), _lib.stream_arg(device)))
    raw = torch.zeros(pages * kv_heads * 4096 + offset, dtype=torch.uint8, device=device)
    data, scales = raw[offset:], torch.zeros(pages, kv_heads, 2, 16, device=device)
    _lib.check(_lib.load().mie_qkv_norm_rope_write_kv8(*common, _lib.ptr(data), kv_heads * 4096, _lib.ptr(scales), *tail,
                                                       pages, 1, 3, 1e-6, _lib.ptr(status), _lib.stream_arg(device)))
    torch.cuda.synchronize()
    assert torch.equal(values.cpu(), values_want)
    # Rounding points are the oracle's; a sum in another order can move the norm by one bf16 step of an entry (2^-8).
    for got, want in ((queries.cpu(), q_want[0].transpose(0, 1)), (keys.cpu(), keys_want)):
        assert (got.float() - want.float()).abs().max() <= 2 ** -7 * want.float().abs().max()
        assert (got != want).float().mean() < 0.05
    pool = data.view(pages, kv_heads, 2, 16, 128).cpu()
    for which, dense in enumerate((keys, values)):
        want_q, want_s = hot_path.quantize_kv_rows(dense.cpu())
        assert torch.equal(pool[:, :, which], want_q)
        assert torch.equal(scales[:, :, which].cpu(), want_s)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols,pad", [(1, 1, 0), (3, 7, 0), (2, 2049, 3), (5, 16384, 8), (4, 151936, 0)])
def test_greedy_tokens_of_logit_rows(dtype, rows, cols, pad, device):
    """The first of the largest values, whatever the alignment; infinities, zeros of both signs, NaN."""

    from mini_inference_engine_b200.engine.kernels.decoder_glue import argmax_rows

    generator = torch.Generator().manual_seed(cols)
    logits = torch.randn(rows, cols + pad, generator=generator).to(dtype)[:, :cols]
    logits[0] = -float("inf")
    if rows > 2:
        logits[1], logits[1, cols // 2], logits[1, cols // 3] = -1.0, 0.0, -0.0
        logits[2, [cols // 2, cols - 1]] = float("inf")
    if rows > 3:
        logits[3, [cols // 3, cols // 2]] = float("nan")
    wide = torch.empty(rows, cols + pad, dtype=dtype, device=device)
    wide[:, :cols] = logits.to(device)
    values = torch.nan_to_num(logits.float(), nan=float("inf"), posinf=3.4e38)  # NaN above infinity
    values = torch.where(logits.isnan(), torch.full_like(values, float("inf")), values)
    want = (values == values.amax(dim=1, keepdim=True)).int().argmax(dim=1)
    assert torch.equal(argmax_rows(wide[:, :cols]).cpu(), want)


@pytest.mark.parametrize("count,offset", [(1, 0), (2, 3), (5, 1), (1023, 2), (4096, 0), (4099, 3)])
def test_soft_cap_of_any_alignment(count, offset, device):
    from mini_inference_engine_b200.engine.kernels.decoder_glue import softcap_

    x = torch.randn(count + offset + 3, generator=torch.Generator().manual_seed(count)) * 50
    x[offset] = float("inf")
    held = x.to(device)
    softcap_(held[offset:offset + count], 30.0)
    want = x.double()
    want[offset:offset + count] = 30.0 * torch.tanh(want[offset:offset + count] / 30.0)
    # tanhf is within 2 units in the last place, the division and the product add half a unit each
    assert ((held.cpu().double() - want).abs() <= 4 * 2 ** -24 * want.abs() * 2).all()


def test_gated_activations_of_any_value(device):
    """SiLU(gate) * up of every bf16 gate, infinities and NaN included: the division's own results."""

    from mini_inference_engine_b200.engine.kernels import fused

    gate = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(torch.bfloat16).view(64, 1024).to(device)
    for factor in (1.0, -0.37):
        up = torch.full_like(gate, factor)
        wide = gate.float()
        want = (wide / (1.0 + torch.exp(-wide))).to(torch.bfloat16) * up
        got = fused.silu_mul(gate, up)
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))
    # The quantised form: an infinite value makes its group's scale infinite.
    gate = torch.ones(1, 256, dtype=torch.bfloat16, device=device)
    gate[0, 5] = float("inf")
    q, scales = torch.empty(1, 256, dtype=torch.uint8, device=device), torch.empty(2, 1, device=device)
    _lib.check(_lib.load().mie_silu_mul(_lib.ptr(gate), _lib.ptr(torch.ones_like(gate)), 256, None, _lib.ptr(q), 256,
                                        _lib.ptr(scales), 1, 1, 256, _lib.stream_arg(device)))
    assert scales[0].item() == float("inf") and 0 < scales[1].item() < 1


@pytest.mark.parametrize("slope", [1.0, 1.702, 1e-6])
def test_clamped_gates_are_ieee_quotients(slope, device):
    """The fp32 form stores the quotient unrounded; gates from subnormal to infinite, no clamp."""

    from mini_inference_engine_b200.engine.kernels.decoder_glue import clamped_glu

    generator = torch.Generator(device=device).manual_seed(5)
    gate = torch.randn(512, 4096, generator=generator, device=device)
    gate[256:] *= torch.exp(torch.linspace(-100, 85, 256, device=device))[:, None]
    gate[0, :4] = torch.tensor([0.0, -0.0, float("inf"), 1e-42], device=device)
    both = torch.cat([gate, torch.zeros_like(gate)], dim=1)
    got = clamped_glu(both, limit=float("inf"), slope=slope, up_offset=1.0)
    want = gate / (1.0 + torch.exp(-slope * gate))
    assert torch.equal(got, want)


def _bf16_values(low: float, high: float, count: int) -> torch.Tensor:
    values = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(torch.bfloat16)
    values = values[(values.float() >= low) & (values.float() <= high)]
    return values[:values.numel() // count * count]


def _units(got: torch.Tensor, want: torch.Tensor) -> torch.Tensor:
    """Errors in units in the last bf16 place."""

    unit = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 7)
    return (got.cpu().double() - want).abs() / unit


@pytest.mark.parametrize("slope", [1.0, 1.702, 0.9, 4.0])
def test_clamped_gates_are_those_of_the_quotient(slope, device):
    """Every bf16 gate whose exponential is finite: half a unit and the fp32 chain's roundings of the exponent (one, which
    |slope g| enlarges), the exponential (two units), the quotient and the product; and the same bits for rows that only
    16-bit accesses fit."""

    from mini_inference_engine_b200.engine.kernels.decoder_glue import clamped_glu

    gates = _bf16_values(-80.0 / slope, 9.0, 8).expand(16, -1)
    ups = torch.randn(gates.shape, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16) * 4
    got = clamped_glu(torch.cat([gates, ups], 1).to(device), limit=7.0, slope=slope, up_offset=1.0)
    z = gates.double().clamp(max=7.0)
    scaled = torch.tensor(slope).double() * z
    want = z / (1.0 + torch.exp(-scaled)) * (ups.double().clamp(-7.0, 7.0) + 1.0)
    assert (_units(got, want) <= 0.5 + 256 * (scaled.abs() + 8) * 2.0 ** -24).all()
    odd = clamped_glu(torch.cat([gates[:, :-3], ups[:, :-3]], 1).to(device), limit=7.0, slope=slope, up_offset=1.0)
    assert torch.equal(odd, got[:, :-3])


def test_gelu_of_any_value(device):
    """Every bf16 value down to where the result is flushed: half a unit and five roundings of the exponent 2 |inner|."""

    from mini_inference_engine_b200.engine.kernels.decoder_glue import gelu

    z = _bf16_values(-9.5, 40.0, 8)
    wide = z.double()
    inner = 0.7978845608028654 * (wide + 0.044715 * wide ** 3)
    want = wide / (1.0 + torch.exp(-2.0 * inner))
    status = torch.zeros(1, dtype=torch.int32, device=device)
    got = gelu(z.view(1, -1).to(device), status=status)[0]
    assert (_units(got, want) <= 0.5 + 256 * (5 * 2 * inner.abs().clamp(max=64) + 8) * 2.0 ** -24).all()
    far = gelu(torch.tensor([[-11.0, -1e30, -float("inf"), float("inf")]], dtype=torch.bfloat16, device=device),
                    status=status)[0].cpu()
    assert far[:2].eq(0).all() and far[2].isnan() and far[3] == float("inf")


# Rows a block: one, several, a last block that is not full; parts of a row; groups of eight and of sixteen lanes (the latter
# up to 3 Mi values); rows of no whole group.
ROW_SHAPES = [(1, 128), (148, 128), (593, 128), (1000, 384), (4100, 1024), (297, 9728), (700, 9728), (5, 12288), (601, 72),
              (1200, 8), (300, 4616)]


@pytest.mark.parametrize("rows,cols", ROW_SHAPES)
def test_gated_rows_of_any_width(rows, cols, device):
    """The division's results (SiLU of every bf16 gate is), and the quantiser's bytes and scales of them."""

    from mini_inference_engine_b200.engine.kernels import fused

    generator = torch.Generator(device=device).manual_seed(rows)
    both = (torch.randn(rows, 2 * cols, generator=generator, device=device) * 3).to(torch.bfloat16)
    wide = both[:, :cols].float()
    want = (wide / (1.0 + torch.exp(-wide))).to(torch.bfloat16) * both[:, cols:]
    assert torch.equal(fused.silu_mul(both[:, :cols], both[:, cols:]), want)
    if cols % 128 == 0:
        q = torch.zeros(rows, cols, dtype=torch.uint8, device=device)
        scales = torch.zeros(cols // 128, rows + 3, device=device)
        _lib.check(_lib.load().mie_silu_mul(_lib.ptr(both), _lib.ptr(both[:, cols:]), 2 * cols, None, _lib.ptr(q), cols,
                                            _lib.ptr(scales), rows + 3, rows, cols, _lib.stream_arg(device)))
        want_q, want_s = sm89_fp8.quantize_sm89_fp8_activation(want)
        assert torch.equal(q, want_q.view(torch.uint8)) and torch.equal(scales[:, :rows].t(), want_s)


@pytest.mark.parametrize("rows,cols", [*ROW_SHAPES, (2000, 37), (10, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gelu_rows_of_any_width(rows, cols, dtype, device):
    """Times a table row for each: the result's rounding to 16 bits, or those of a few fp32 operations and of 1 + tanh."""

    from mini_inference_engine_b200.engine.kernels.decoder_glue import gelu

    generator = torch.Generator().manual_seed(cols)
    x, table = torch.randn(rows, cols, generator=generator).to(dtype), torch.randn(7, cols, generator=generator).to(dtype)
    ids = torch.arange(rows) % 7
    status = torch.zeros(1, dtype=torch.int32, device=device)
    got = gelu(x.to(device), ids=ids.to(device), table=table.to(device), status=status).cpu().double()
    z = x.double()
    want = z / (1.0 + torch.exp(-2.0 * 0.7978845608028654 * (z + 0.044715 * z ** 3))) * table.double()[ids]
    bound = want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19)
    assert ((got - want).abs() <= bound + (z * table.double()[ids]).abs() * 2.0 ** -21).all() and int(status.item()) == 0


@pytest.mark.parametrize("rows,cols", [(1400, 8), (9500, 128), (2700, 1024), (1500, 1792), (700, 2560), (310, 4096), (200, 8192)])
def test_norm_rows_past_the_resident_blocks(rows, cols, device):
    """Blocks that go from row to row: residual sum, norm and e4m3.  The sum's order can move a normed value by one bf16 step
    (2^-7 of it at most); the product with the weight is rounded on both sides, half a step each: 2^-6 in all."""

    generator = torch.Generator().manual_seed(cols)
    x, residual, weight = (torch.randn(n, cols, generator=generator).to(torch.bfloat16).to(device) for n in (rows, rows, 1))
    summed, out = torch.empty_like(x), torch.empty_like(x)
    q, scales = torch.zeros(rows, cols, dtype=torch.uint8, device=device), torch.zeros(max(1, cols // 128), rows, device=device)
    fits = cols % 128 == 0
    _lib.check(_lib.load().mie_rms_norm(_lib.ptr(x), cols, _lib.ptr(residual), _lib.ptr(summed), _lib.ptr(weight),
                                        _lib.ptr(out), _lib.ptr(q) if fits else None, cols, _lib.ptr(scales), rows, rows,
                                        cols, 1e-6, _lib.stream_arg(device)))
    assert torch.equal(summed, x + residual)
    want = hot_path.rms_norm(summed.cpu(), weight[0].cpu(), 1e-6).float()
    assert ((out.cpu().float() - want).abs() <= 2.0 ** -6 * want.abs()).all()
    assert (out.cpu().float() != want).float().mean() < 0.02
    if fits:
        want_q, want_s = sm89_fp8.quantize_sm89_fp8_activation(out)
        assert torch.equal(q, want_q.view(torch.uint8)) and torch.equal(scales.t(), want_s)
