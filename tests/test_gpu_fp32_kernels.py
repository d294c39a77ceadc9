"""The float32 product kernels give, bit for bit, what the plain kernels give: an operand that does not start
on 16 bytes goes to the plain kernel, whose additions run in the same order."""
import pytest
import torch

from test_gpu_kernels import rnd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def off_by_one(x):
    """The same numbers one float32 behind a 16-byte boundary."""
    held = torch.empty(x.numel() + 4, device=DEV)
    y = held[1:1 + x.numel()].view(x.shape)
    y.copy_(x)
    assert y.data_ptr() % 16 == 4
    return y


# rows at and around the places where the kernel changes (1, 2, 4, 8, 16 | tiles); columns at and around 8, 32, 64, 128, the
# changes of the few-row plan (16 and 32 columns an SM) and a wide output; K around the chunks of 32 and 128
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 70, 129, 300])
@pytest.mark.parametrize("N,K", [(1, 4), (8, 96), (40, 124), (65, 132), (130, 224), (2376, 260), (4744, 128), (9001, 36)])
def test_float32_product_adds_in_the_plain_kernels_order(M, N, K):
    from purhie_b200.csrc import ops
    x, w = rnd(M, K, seed=M), rnd(N, K, seed=N)
    out, plain = torch.full((M, N), float("nan"), device=DEV), torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_simple(x, w, out)
    ops.gemm_simple(off_by_one(x), w, plain)
    assert torch.equal(out, plain)
    # K products, each exact inside one rounded multiply-add: at most K half units in the last place of the sum of magnitudes
    bound = K * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)
    assert ((out.double() - x.double() @ w.double().T).abs() <= bound).all()
