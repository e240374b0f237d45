"""Products of a few rows with a weight matrix (ktk_linear_rows) against fp64, and what the decoder layer sends there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("n, k", [(1, 8), (7, 72), (64, 2048), (770, 512), (5, 2056), (33, 4096)])
def test_products(cuda_device, dtype, rows, n, k):
    # fewer columns than a CTA takes, inner sizes under, at and over a step of a CTA's threads.  Bound: sums of k products of size one in
    # fp32, k 2^-24 at the very most, and the rounding of the result
    from kinetics_b200 import ops
    g = torch.Generator().manual_seed(rows * n + k)
    put = lambda *s: torch.randn(*s, generator=g).to(dtype).to(cuda_device)
    x, w, w2, b, res = put(rows, k), put(n, k), put(n, k), put(n), put(rows, n)
    tol = dict(rtol=1e-5, atol=1e-5 * k ** 0.5) if dtype == torch.float32 else dict(rtol=8e-3, atol=1e-5 * k ** 0.5)
    d = lambda t: t.double()
    y = d(x) @ d(w).t()
    close = lambda got, want: torch.testing.assert_close(got.double(), want, **tol)
    close(ops.linear_rows(x, w), y)
    close(ops.linear_rows(x, w, bias=b), y + d(b))
    close(ops.linear_rows(x, w, bias=b, residual=res), y + d(b) + d(res))
    x, u = x * k ** -0.5, d(x * k ** -0.5) @ d(w2).t()
    y = d(x) @ d(w).t()
    torch.testing.assert_close(ops.linear_rows(x, w, w2=w2).double(), torch.nn.functional.silu(y) * u,
                               rtol=1e-5 if dtype == torch.float32 else 8e-3, atol=1e-5)


def test_refused(cuda_device):
    from kinetics_b200 import ops
    z = lambda *s: torch.zeros(*s, device=cuda_device)
    for x, w in ((z(17, 8), z(4, 8)), (z(4, 16), z(4, 8)), (z(4, 12), z(4, 12))):
        with pytest.raises((ValueError, RuntimeError)):
            ops.linear_rows(x, w)
    with pytest.raises(RuntimeError):
        ops.linear_rows(z(33)[1:].view(4, 8), z(4, 8))       # starts between two 16-byte pieces


def test_a_hooked_layer_is_called(cuda_device):
    # a hook on a projection sees its call, and what it returns is what goes on
    from kinetics_b200 import layers
    lin = torch.nn.Linear(64, 32, device=cuda_device).requires_grad_(False)
    x = torch.randn(4, 64, device=cuda_device)
    assert layers._by_rows(x, lin)
    plain = layers._linear(lin, x)
    torch.testing.assert_close(plain, lin(x), rtol=1e-5, atol=1e-5)
    handle = lin.register_forward_hook(lambda m, i, o: o + 1)
    assert not layers._by_rows(x, lin)
    torch.testing.assert_close(layers._linear(lin, x), plain + 1, rtol=1e-5, atol=1e-5)
    handle.remove()
    assert not layers._by_rows(x.half(), lin) and not layers._by_rows(x.t(), lin)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not layers._by_rows(x, lin)


def test_a_bias_that_is_not_contiguous_stays_with_the_library(cuda_device):
    from kinetics_b200 import layers
    lin = torch.nn.Linear(64, 32, device=cuda_device).requires_grad_(False)
    x, plain = torch.randn(4, 64, device=cuda_device), lin.bias.detach().clone()
    lin.bias = torch.nn.Parameter(torch.stack((plain, plain + 1), dim=1)[:, 0], requires_grad=False)
    assert not lin.bias.is_contiguous()
    want = x.double() @ lin.weight.double().t() + plain.double()
    torch.testing.assert_close(layers._linear(lin, x).double(), want, rtol=1e-5, atol=1e-5)
    with pytest.raises(RuntimeError):                        # refused as the library refuses it
        layers._linear(lin, torch.randn(4, 72, device=cuda_device))
