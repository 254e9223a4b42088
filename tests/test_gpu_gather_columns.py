"""The column gather of W46Linear against torch's index_select and addition: same bits."""
import pytest
import torch

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
