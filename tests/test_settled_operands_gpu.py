"""What a kernel reads before its wait for the kernels ahead, it reads only where the caller has said that none of those writes it."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows", [1, 16])
@pytest.mark.parametrize("late", ["weights", "input"])
def test_a_head_product_of_what_was_made_just_ahead(rows, late):
    """Its weights (no promise is given) or its input (the weights are settled) come from the launch before, written last after a long
    product: every one of them is seen."""
    g = torch.Generator(device=DEV).manual_seed(rows)
    heads, k, n, inner = 2, 128, 512, 8192
    strides = dict(n_tokens=rows, n_heads=heads, k=k, n=n, in_strides=(heads * k, k), w_strides=(k * n, 1, k), out_strides=(heads * n, n))
    x = torch.randn(rows, heads * k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(heads * n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    made = w if late == "weights" else x
    left = torch.randn(made.shape[0], inner, generator=g, device=DEV).bfloat16()
    right = (torch.randn(made.shape[1], inner, generator=g, device=DEV) * inner ** -0.5).bfloat16()
    first, again = torch.empty(rows, heads * n, device=DEV).bfloat16(), torch.empty(rows, heads * n, device=DEV).bfloat16()
    for _ in range(5):
        made.fill_(float("nan"))
        K.linear(left, right, None, made)
        K.head_linear(x, w, first, w_settled=late == "input", **strides)
        K.head_linear(x, w, again, w_settled=True, **strides)  # all of it long there: the same sums
        assert first.isfinite().all() and torch.equal(first, again)
        want = torch.einsum("thk,hnk->thn", x.view(rows, heads, k).double(), w.view(heads, n, k).double()).reshape(rows, -1)
        # a bfloat16 rounding, and float32 sums of 128 products of order up to 12
        assert ((first.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-3).all()
