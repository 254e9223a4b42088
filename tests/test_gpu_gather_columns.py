"""The column gather of W46Linear against torch's index_select and addition: same bits."""
import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 8), (3, 256), (5, 1032), (201, 4096), (4, 1024), (262145, 8)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_same_as_index_select(m, n, with_bias):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    c = torch.randn((m, n), generator=gen, device="cuda").half()
    c[0, 0], c[-1, -1] = float("inf"), float("nan")
    src = torch.randperm(n, generator=gen, device="cuda")
    bias = torch.randn(n, generator=gen, device="cuda").half() if with_bias else None
    expect = c.index_select(1, src)
    if with_bias:
        expect = expect + bias
    got = api.gather_columns(c, src, bias)
    assert torch.equal(got.isnan(), expect.isnan())
    assert torch.equal(got.nan_to_num(7.0), expect.nan_to_num(7.0))


def test_forms_that_keep_the_torch_operations():
    c = torch.randn((4, 20), device="cuda").half()                              # no multiple of 8
    src = torch.randperm(20, device="cuda")
    assert torch.equal(api.gather_columns(c, src), c[:, src])
    c = torch.randn((4, 64), device="cuda").half()
    src = torch.arange(65, device="cuda")[1:] - 1
    bias = torch.nn.Parameter(torch.randn(64, device="cuda").half())
    y = api.gather_columns(c, src, bias)                                        # a trainable bias keeps its graph
    y.float().sum().backward()
    assert torch.equal(bias.grad, torch.full_like(bias, 4.0))
    assert api.gather_columns(c, src, bias.detach().float()).dtype == torch.float32
    assert torch.equal(api.gather_columns(c, torch.arange(-1, 64, device="cuda")[1:]), c)      # indices off the 16-byte grid
    assert torch.equal(api.gather_columns(c, src[:8]), c[:, :8])                # fewer columns


def test_bias_under_function_transforms():
    """Forward-mode derivatives of the bias, and maps over it, go through the torch operations."""
    from torch.autograd import forward_ad

    gen = torch.Generator(device="cuda").manual_seed(5)
    c = torch.randn((4, 64), generator=gen, device="cuda").half()
    src = torch.randperm(64, generator=gen, device="cuda")
    bias, tangent = (torch.randn(64, generator=gen, device="cuda").half() for _ in range(2))
    plain = c.index_select(1, src) + bias
    with forward_ad.dual_level():
        y = forward_ad.unpack_dual(api.gather_columns(c, src, forward_ad.make_dual(bias, tangent)))
        assert torch.equal(y.primal, plain) and y.tangent is not None and torch.equal(y.tangent, tangent.expand(4, 64))
        z = forward_ad.unpack_dual(api.gather_columns(forward_ad.make_dual(c, c), src, bias))
        assert torch.equal(z.tangent, c.index_select(1, src))
        assert forward_ad.unpack_dual(api.gather_columns(c, src, bias)).tangent is None
    primal, pushed = torch.func.jvp(lambda b: api.gather_columns(c, src, b), (bias,), (tangent,))
    assert torch.equal(primal, plain) and torch.equal(pushed, tangent.expand(4, 64))
    many = torch.stack([bias, tangent, bias + tangent])
    mapped = torch.func.vmap(lambda b: api.gather_columns(c, src, b))(many)
    assert torch.equal(mapped, torch.stack([api.gather_columns(c, src, b) for b in many.unbind()]))
    primal, pushed = torch.func.jvp(torch.func.vmap(lambda b: api.gather_columns(c, src, b)), (many,), (many,))
    assert torch.equal(primal, mapped) and torch.equal(pushed, many[:, None].expand(3, 4, 64))
    grad = torch.func.grad(lambda b: api.gather_columns(c, src, b).float().sum())(bias)
    assert torch.equal(grad, torch.full_like(bias, 4.0))

    layer = fm.W46Linear((torch.randn((256, 128), generator=gen, device="cuda") * 0.02).half(), 64, 128, torch.zeros(256)).cuda()
    x = torch.randn((3, 128), generator=gen, device="cuda").half()
    biases = torch.randn((2, 256), generator=gen, device="cuda").half()
    ordered = fm.set_ordered_sums(True)
    try:
        got = torch.func.vmap(lambda b: torch.func.functional_call(layer, {"bias": b}, (x,)))(biases)
        assert torch.equal(got, layer(x)[None] + biases[:, None])
    finally:
        fm.set_ordered_sums(ordered)
