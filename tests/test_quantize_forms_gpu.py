"""The two forms of the quantisation (a cluster per segment, two passes) at the sizes where one takes over
from another or a piece is not full: same bytes and scales as plain torch."""
import time

import pytest
import torch

from cutlass_flash_atten_fp8_b200 import quantize_e4m3

pytestmark = pytest.mark.gpu


def check(x, per_head):
    y, descale = quantize_e4m3(x, per_head=per_head)
    amax = (x.abs().amax(dim=(2, 3), keepdim=True) if per_head else x.abs().amax()).float()
    top = torch.tensor(448.0, device=x.device)
    want = (x.float() * torch.div(top, amax)).to(torch.float8_e4m3fn)
    assert torch.equal(y.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(descale, torch.div(amax.flatten(), top))


# elements of a lone tensor: one vector less and more than a thread's registers hold (128 x 8 and 512 x 8
# vectors of 8), one more than a cluster's (8 x 512 x 8), and sizes of one vector more than a power of two or a full grid
# up to more than stays in L2
@pytest.mark.parametrize("n", [1, 7, 9, 8191, 8200, 32768 + 8, 262144, 262144 + 13, 9699328 + 9, 24248320 + 8, 24248320 * 2 + 3,
                               192 * 2 ** 19 + 11])
def test_lone_tensors(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, generator=g, device="cuda").to(torch.float16 if n % 2 else torch.bfloat16)
    for at in {0, n // 2, n - 1}:                 # the largest value at either end and in the middle
        z = x.clone()
        z[at] = -9.0
        check(z, False)


@pytest.mark.parametrize("shape", [(2, 3, 1, 32), (4, 8, 64, 128), (3, 4, 2048, 128), (3, 4, 2056, 128), (2, 2, 4096, 128), (2, 6, 6144, 128),
                                   (2, 6, 6152, 128), (1, 11, 6144, 128), (16, 130, 16, 64)])
def test_segments(shape):
    g = torch.Generator(device="cuda").manual_seed(shape[2])
    x = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    x[0, 0, -1, -1] = 11.0
    check(x, True)


def test_lone_zeros_and_nan():
    for n in (1000, 10 ** 6, 2 * 10 ** 8):
        x = torch.zeros(n, device="cuda", dtype=torch.float16)
        y, descale = quantize_e4m3(x)
        assert not bool(y.view(torch.uint8).any()) and float(descale) == 1.0
        x[n // 3], x[n // 2] = float("nan"), 2.0
        y, descale = quantize_e4m3(x)
        assert bool(y.float()[n // 3].isnan()) and float(y.float()[n // 2]) == 448.0 and abs(float(descale) * 224.0 - 1.0) < 1e-6


@pytest.mark.parametrize("shape,per_head", [((1, 1, 1000, 64), False), ((1, 16, 2048, 128), False), ((1, 32, 8192, 128), False),
                                            ((4, 32, 2048, 128), True), ((4, 32, 4096, 128), True), ((1, 4, 8192, 128), True)])
def test_a_long_kernel_elsewhere_is_not_waited_for(shape, per_head):
    # one block that keeps a little of one SM for about 0.2 s on another stream; in a serving process it could be
    # waiting for this stream
    x = torch.randn(shape, device="cuda").to(torch.float16)
    quantize_e4m3(x, per_head=per_head)
    torch.cuda.synchronize()
    side, asleep, done = torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)
        asleep.record()
    time.sleep(0.01)
    quantize_e4m3(x, per_head=per_head)
    done.record()
    done.synchronize()
    assert not asleep.query()
    torch.cuda.synchronize()
