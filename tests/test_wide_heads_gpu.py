"""Head dims over 128 (one query tile per CTA, scores of a 128-key tile in one product, four score buffers
and four softmax warps per row group): key counts around one to six sub-blocks of 64, where a product
covers one sub-block or two, a warp has no sub-block at all, and buffers are used for the second time;
several items per CTA.  Tolerance: the rounding of P to e4m3, as in test_parity_gpu."""
import math

import pytest
import torch

from cutlass_flash_atten_fp8_b200 import check_status, flash_attention_v2_cutlass
from oracle.attention_oracle import error_metrics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [160, 192, 224, 256])
@pytest.mark.parametrize("layout", ["natural", "transposed"])
@pytest.mark.parametrize("causal", [False, True])
def test_sub_block_counts(D, layout, causal):
    d = torch.device("cuda", 0)
    for Sq, Sk in [(65, 16), (128, 64), (200, 80), (128, 128), (300, 192), (257, 208), (128, 256), (384, 336), (500, 384), (129, 640)]:
        g = torch.Generator().manual_seed(Sq + Sk + D)
        q, k, v = ((torch.randn(20, 4, s, D, generator=g) * f).to(torch.float8_e4m3fn).to(d) for s, f in ((Sq, 2.0), (Sk, 1.0), (Sk, 1.0)))
        scale = 1 / math.sqrt(D)
        vv = v if layout == "natural" else v.transpose(2, 3).contiguous()
        out, lse = flash_attention_v2_cutlass(q, k, vv, causal, scale, v_layout=layout, return_lse=True)
        check_status(d)
        s = q.float() @ k.float().transpose(2, 3) * scale
        if causal:
            s = s.masked_fill(torch.arange(Sk, device=d).unsqueeze(0) > torch.arange(Sq, device=d).unsqueeze(1), float("-inf"))
        m = error_metrics(out.cpu(), (torch.softmax(s, -1) @ v.float()).cpu())
        assert m["rel_l2"] <= 3e-2, (Sq, Sk, m)
        assert float((lse - torch.logsumexp(s, -1)).abs().max()) <= 2e-3, (Sq, Sk)
