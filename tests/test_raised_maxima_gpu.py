"""Row maxima that are raised in every sub-block of 64 keys: scores climb by eight per sub-block for half of
the rows and fall for the others, so O is rescaled (by e^-8) before nearly every product.  A sub-block whose
contribution misses the factor would outweigh the true result.  Many more slices than SMs and one or two query
tiles, so that items start cold, with V arriving last.  Tolerance: the rounding of P to e4m3, as in test_parity_gpu."""
import pytest
import torch

from cutlass_flash_atten_fp8_b200 import check_status, flash_attention_v2_cutlass
from oracle.attention_oracle import error_metrics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 64, 96, 128, 160, 256])
@pytest.mark.parametrize("Sq,Sk,v_layout", [(128, 192, "transposed"), (100, 330, "natural"), (256, 1024, "transposed")])
def test_contributions_before_a_raise_are_scaled(D, Sq, Sk, v_layout):
    dev, n = torch.device("cuda", 0), 449
    g = torch.Generator(device=dev).manual_seed(D + Sk)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev)
    sign = torch.where(rand(1, n, Sq, 1) > 0, 1.0, -1.0)
    q = (sign * (1 + 0.1 * rand(1, n, Sq, D))).to(torch.float8_e4m3fn)
    climb = (torch.arange(Sk, device=dev) // 64).float().view(1, 1, Sk, 1)
    k = (climb + 0.25 * rand(1, n, Sk, D)).to(torch.float8_e4m3fn)
    v = rand(1, n, Sk, D).to(torch.float8_e4m3fn)
    scale = 8.0 / D
    given = v if v_layout == "natural" else v.transpose(2, 3).contiguous()
    s = (q.double() @ k.double().transpose(2, 3)) * scale
    want, want_lse = torch.softmax(s, -1) @ v.double(), torch.logsumexp(s, -1)
    for _ in range(3):
        out, lse = flash_attention_v2_cutlass(q, k, given, False, scale, v_layout=v_layout, return_lse=True)
        check_status(dev)
        assert error_metrics(out, want)["rel_l2"] <= 3e-2
        worst = (out.double() - want).norm(dim=-1) / want.norm(dim=-1)
        # 64 or fewer keys share a row's weight, each off by 2^-4 at most and independently: a few hundredths; a
        # missing factor makes it about 1
        assert float(worst.max()) <= 0.25, float(worst.max())
        assert float((lse.double() - want_lse).abs().max()) <= 1e-4 * float(want_lse.abs().max())
