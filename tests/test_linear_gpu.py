"""bf16 projections of decode-sized batches against the product in 64 bits."""

from __future__ import annotations

import pytest
import torch

from mini_inference_engine_b200.engine.kernels.linear import linear, linear_supported

pytestmark = pytest.mark.gpu

# Weight rows and columns around the tiles of both kernels (16 and 128 rows, units of 64 columns, K cut in up to 8).
SHAPES = [(1, 8), (16, 64), (17, 72), (127, 520), (129, 256), (2048, 2048), (8200, 512), (2112, 4096), (300, 6152)]


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("kernel", [1, 2])
def test_product_against_64_bits(n, k, m, kernel, device):
    if kernel == 1 and m > 32:
        pytest.skip("the register kernel takes up to 32 rows")
    torch.manual_seed(n * 31 + k + m)
    # Rows of a wider buffer and a nonsense tail past k: the kernels must honour the strides.
    x = torch.full((m, k + 24), float("nan"), dtype=torch.bfloat16, device=device)[:, :k]
    w = torch.full((n, k + 8), float("nan"), dtype=torch.bfloat16, device=device)[:, :k]
    x.copy_(torch.randn(m, k, device=device))
    w.copy_(torch.randn(n, k, device=device) / k ** 0.5)
    bias = torch.randn(n, device=device).to(torch.bfloat16) if m % 2 else None
    status = torch.zeros(1, dtype=torch.int32, device=device)
    assert linear_supported(x, w, bias)
    out = linear(x, w, bias, status=status, kernel=kernel)
    exact = x.double() @ w.double().t() + (0.0 if bias is None else bias.double())
    # One rounding to bf16 (2^-9 of the value) of sums whose fp32 error is below k 2^-24 of the terms' magnitude.
    bound = exact.abs() * 2.0 ** -8 + k * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t()) + 1e-30
    assert bool(((out.double() - exact).abs() <= bound).all())
    assert int(status.item()) == 0


def test_infinities_and_nans_stay_where_they_belong(device):
    for kernel, m in ((1, 5), (2, 40)):
        x = torch.ones(m, 128, dtype=torch.bfloat16, device=device)
        w = torch.ones(64, 128, dtype=torch.bfloat16, device=device)
        x[1, 3], w[7, 70] = float("inf"), float("nan")
        status = torch.zeros(1, dtype=torch.int32, device=device)
        out = linear(x, w, status=status, kernel=kernel).float()
        assert bool(out[:, 7].isnan().all())
        rest = torch.cat([out[:, :7], out[:, 8:]], dim=1)
        assert bool((rest[1] == float("inf")).all()) and bool((rest[0] == 128).all())


def test_what_the_kernels_do_not_take_goes_to_the_library(device):
    x, w = torch.randn(4, 12, device=device), torch.randn(6, 12, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    for a, b in ((x, w), (x.bfloat16(), w.bfloat16()), (x[:0].bfloat16(), w.bfloat16())):
        assert not linear_supported(a, b)
        torch.testing.assert_close(linear(a, b, status=status), torch.nn.functional.linear(a, b))


@pytest.mark.parametrize("m,n,k", [(3, 4096, 512), (20, 12288, 4096)])
def test_weights_written_by_a_queued_kernel(m, n, k, device):
    """``MIE_LINEAR_NO_WEIGHT_PREFETCH``: the weights are read after the kernel of this library that writes them."""

    from mini_inference_engine_b200 import _lib
    from mini_inference_engine_b200.engine.kernels.decoder_glue import gelu

    generator = torch.Generator(device=device).manual_seed(m)
    sources = [torch.randn(n, k, generator=generator, device=device).bfloat16() for _ in range(2)]
    x = torch.randn(m, k, generator=generator, device=device).bfloat16()
    status, out = torch.zeros(1, dtype=torch.int32, device=device), torch.empty(m, n, dtype=torch.bfloat16, device=device)

    def step(source, wait):
        w = gelu(source)
        if wait:
            torch.cuda.synchronize()
        _lib.check(_lib.load().mie_linear(_lib.ptr(x), k, _lib.ptr(w), k, None, _lib.ptr(out), n, m, n, k, 4,
                                          _lib.ptr(status), _lib.stream_arg(device)))
        return out.clone()

    want = [step(source, True) for source in sources]
    for i in range(20):
        assert torch.equal(step(sources[i % 2], False), want[i % 2])
    assert int(status.item()) == 0


@pytest.mark.parametrize("m,n,k,kernel", [(8, 4096, 2048, 1), (8, 2040, 4096, 2), (8, 680, 12288, 2), (16, 512, 2048, 1),
                                          (16, 240, 4096, 2)])
def test_which_kernel_takes_a_product(m, n, k, kernel, device):
    """Long sums belong to the kernel that cuts K.  The two add in different orders, and the halves of every sum nearly
    cancel, so the bits tell them apart."""

    generator = torch.Generator(device=device).manual_seed(n)
    x = torch.randn(m, k, generator=generator, device=device).bfloat16()
    w = torch.randn(n, k, generator=generator, device=device).bfloat16()
    w[:, k // 2:] = -w[:, :k // 2]
    x[:, k // 2:] = x[:, :k // 2] * (1 + 2.0 ** -7)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    picked, named, other = (linear(x, w, status=status, kernel=which) for which in (0, kernel, 3 - kernel))
    assert torch.equal(picked, named) and not torch.equal(picked, other)


def test_whatever_the_library_product_takes(device):
    """Shapes and strides that the kernels do not take: as ``torch.nn.functional.linear``, before and after."""

    generator = torch.Generator(device=device).manual_seed(1)
    x, w = (torch.randn(r, 64, generator=generator, device=device).bfloat16() for r in (4, 32))
    bias, status = torch.randn(32, device=device).bfloat16(), torch.zeros(1, dtype=torch.int32, device=device)
    for a, b, c in ((x.view(2, 2, 64), w, None), (x[0], w, bias), (x[:1].expand(3, 64), w, bias), (x, w[:1].expand(5, 64), None),
                    (x, w[0], None), (x.t().contiguous().t(), w, None), (x, w[:0], None), (x[:, :0], w[:, :0], None),
                    (x, w, bias.float().bfloat16().expand(32)), (x.as_strided((4, 64), (8, 1)), w, None)):
        torch.testing.assert_close(linear(a, b, c, status=status), torch.nn.functional.linear(a, b, c))
    weight = w.clone().requires_grad_()
    linear(x, weight, bias, status=status).sum().backward()
    torch.testing.assert_close(weight.grad, x.sum(0).expand(32, 64), rtol=2 ** -7, atol=2 ** -6)


def test_operands_that_do_not_belong_together_are_refused(device):
    """A weight of other columns (its rows would be read past their end), a bias of another length."""

    x, w = torch.randn(4, 64, device=device).bfloat16(), torch.randn(32, 48, device=device).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device=device)
    for a, b, c in ((x, w, None), (x[:, :48], w, torch.zeros(31, device=device).bfloat16()), (x[:, :48], w.cpu(), None)):
        assert not linear_supported(a, b, c)
        with pytest.raises(RuntimeError):
            linear(a, b, c, status=status)
