"""Kernels that may start before their predecessor has finished: a chain in which every launch reads what
the one before wrote, into buffers that are used again, gives the same bits as with a synchronisation
after every launch.  Small grids (SMs free for the successor) and full ones, in a stream and in a graph."""
import pytest
import torch

from cutlass_flash_atten_fp8_b200 import flash_attention_v2_cutlass, quantize_e4m3

pytestmark = pytest.mark.gpu


def chain(x, out, steps, per_head, sync):
    pause = torch.cuda.synchronize if sync else (lambda: None)
    for i in range(steps):
        y, d = quantize_e4m3(x if i == 0 else out, per_head=per_head)
        pause()
        rows = y[:, :, :3].contiguous()
        few = flash_attention_v2_cutlass(rows, y, y, False, 0.1, v_layout="natural", descale_q=d, descale_k=d, descale_v=d)[0]
        pause()
        flash_attention_v2_cutlass(y, y, y, i % 2 == 1, 0.1, v_layout="natural", descale_q=d, descale_k=d, descale_v=d, out=out)
        pause()
    return few


@pytest.mark.parametrize("shape", [(1, 2, 100, 64), (2, 8, 777, 128), (8, 32, 640, 64), (1, 4, 1300, 256)])
@pytest.mark.parametrize("per_head", [False, True])
def test_chain_of_dependent_launches(shape, per_head):
    x = torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").to(torch.float16)
    want, out = torch.empty_like(x), torch.empty_like(x)
    few = chain(x, want, 6, per_head, True).clone()
    for _ in range(3):
        got = chain(x, out, 6, per_head, False)
        assert torch.equal(out, want) and torch.equal(got, few)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(x, out, 6, per_head, False)
    out.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(got, few)
