"""TFT backward of more batch items than SMs, 16- and 32-wide heads: two items to an SM, V and every head's K through one buffer.  Key counts that are
no multiple of four, one and several row tiles and heads, a last tile of one row; against the fp64 oracle at the bound of the other kernels."""
import pytest

from test_tft_split_gpu import cuda, forward_and_backward  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_attn_grad", [False, True])
@pytest.mark.parametrize("B,H,Nq,Nk,d", [(149, 2, 50, 61, 32), (151, 3, 24, 192, 16), (150, 1, 25, 33, 32), (149, 1, 1, 1, 16), (300, 4, 7, 130, 16)])
def test_two_items_to_an_sm(cuda, B, H, Nq, Nk, d, with_attn_grad):  # noqa: F811
    forward_and_backward(cuda, B, H, Nq, Nk, d, with_attn_grad, with_mask=True)


@pytest.mark.parametrize("B,H,Nq,Nk,d", [(149, 2, 30, 61, 32), (150, 3, 24, 190, 16)])
def test_without_a_mask(cuda, B, H, Nq, Nk, d):  # noqa: F811
    forward_and_backward(cuda, B, H, Nq, Nk, d, True, with_mask=False)
