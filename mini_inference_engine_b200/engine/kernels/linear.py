"""bf16 projections of decode-sized batches (``csrc/linear.cu``); everything else goes to the library product."""

from __future__ import annotations

import torch

from ... import _lib

MAX_ROWS = 128  # MIE_LINEAR_MAX_ROWS


def linear_supported(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None) -> bool:
    """Whether ``mie_linear`` takes the product: a few bf16 rows that do not overlap, 16-byte aligned, whole 16-byte
    groups, nothing that autograd follows."""

    if not (x.ndim == weight.ndim == 2 and 0 < x.shape[0] <= MAX_ROWS and x.dtype == weight.dtype == torch.bfloat16):
        return False
    (n, k), operands = weight.shape, [x, weight]
    if bias is not None:
        operands.append(bias)
        if bias.dtype != torch.bfloat16 or tuple(bias.shape) != (n,) or not bias.is_contiguous():
            return False
    return bool(x.is_cuda and x.shape[1] == k and n > 0 and k > 0 and k % 8 == 0
                and all(t.device == x.device for t in operands)
                and x.stride(1) == weight.stride(1) == 1 and x.stride(0) >= k and weight.stride(0) >= k
                and x.stride(0) % 8 == 0 and weight.stride(0) % 8 == 0
                and x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0
                and not (torch.is_grad_enabled() and any(t.requires_grad for t in operands)))


def prefers_own_kernel(rows: int, n: int, k: int) -> bool:
    """Where the kernels of ``csrc/linear.cu`` beat the library product inside a launch chain (a norm before each
    product, weights from HBM; us, library / this): up to 8 rows everywhere (2048 x 2048 9.8 / 5.2, 4096 x 12288
    37.7 / 21.1; at worst even, 12288 x 2048 of 8 rows 13.2 / 13.4); up to 16 rows also small outputs (4096 x 2048
    8.9 / 7.8, but 16384 x 2048 16.3 / 17.0); up to 64 rows long sums (4096 x 12288 28.7 / 24.9, 256 x 4096 10.6 / 8.0,
    12288 x 4096 24.9 / 22.7, but 4096 x 2048 7.9 / 9.2), where the library cuts K too little.  At 128 rows reading the
    activations once per weight tile costs more than it saves (7.6 / 14)."""

    return rows <= 8 or (rows <= 16 and n <= 4096) or (rows <= 64 and k >= 4096)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None, *, status: torch.Tensor,
           kernel: int = 0) -> torch.Tensor:
    """``x [rows, k] @ weight [n, k]^T (+ bias)`` for weights that no queued kernel of this library writes (a model's
    parameters).  ``kernel``: 0 picks, 1 / 2 name one of the two kernels."""

    if not linear_supported(x, weight, bias):
        return torch.nn.functional.linear(x, weight, bias)
    (rows, k), n = x.shape, int(weight.shape[0])
    if not (kernel or prefers_own_kernel(rows, n, k)):
        return torch.nn.functional.linear(x, weight, bias)
    out = torch.empty(rows, n, dtype=x.dtype, device=x.device)
    _lib.check(_lib.load().mie_linear(_lib.ptr(x), x.stride(0), _lib.ptr(weight), weight.stride(0), _lib.ptr(bias),
                                      _lib.ptr(out), n, rows, n, k, kernel, _lib.ptr(status),
                                      _lib.stream_arg(x.device)))
    return out


__all__ = ["MAX_ROWS", "linear", "linear_supported", "prefers_own_kernel"]
