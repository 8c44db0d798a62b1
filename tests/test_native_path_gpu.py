"""The package's operators through the compiled module and through ctypes: the same parameter blocks, hence
the same bits."""
import pytest
import torch

from cutlass_flash_atten_fp8_b200 import api, check_status, flash_attention_v2_cutlass, quantize_e4m3

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.fixture
def both_ways(monkeypatch):
    """call(f) -> (result of f through the compiled module, result through ctypes)"""
    native = api._native()
    assert native, "build the module first: python -m cutlass_flash_atten_fp8_b200.build --binding"
    taken = []

    class Counting:                                      # what the module did not take would go through ctypes as well
        def __getattr__(self, name):
            def through(*a):
                r = getattr(native, name)(*a)
                taken.append(r)
                return r
            return through

    def call(f):
        monkeypatch.setattr(api, "_native_module", Counting())
        taken.clear()
        one = f()
        assert len(taken) == 1 and taken[0] is not None
        monkeypatch.setattr(api, "_native_module", False)
        two = f()
        check_status(DEV)
        return one, two
    return call


def same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.shape == y.shape and x.dtype == y.dtype and x.device == y.device
        assert torch.equal(x.reshape(-1).view(torch.uint8), y.reshape(-1).view(torch.uint8))


def tensors(B, H, Hk, Sq, Sk, D, v_layout, dtype=torch.float8_e4m3fn):
    g = torch.Generator(device=DEV).manual_seed(Sq + Sk + D)
    q, k, v = (torch.randn(B, h, s, D, generator=g, device=DEV).to(dtype) for h, s in ((H, Sq), (Hk, Sk), (Hk, Sk)))
    return q, k, v if v_layout == "natural" else v.transpose(2, 3).contiguous()


def scales(n, seed):
    return 0.5 + torch.rand(n, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


# shapes: equal lengths, grouped heads with other lengths (ragged where the layout allows), few query rows
@pytest.mark.parametrize("shape,v_layout", [((2, 4, 4, 256, 256, 64), "transposed"), ((2, 6, 2, 77, 208, 128), "transposed"),
                                            ((2, 6, 2, 65, 333, 128), "natural"), ((3, 8, 2, 1, 700, 96), "natural"),
                                            ((1, 2, 1, 130, 97, 256), "natural")])
@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("causal", [False, True])
def test_attention(both_ways, shape, v_layout, dtype, causal):
    B, H, Hk, Sq, Sk, D = shape
    q, k, v = tensors(*shape, v_layout, dtype)
    for descale in ({}, {"descale_q": scales(1, 1)}, {"descale_" + n: scales(1, i) for i, n in enumerate("qkv")},
                    {"descale_q": scales(B * H, 1), "descale_k": scales(B * Hk, 2), "descale_v": scales(B * Hk, 3)}):
        for kw in ({}, {"return_lse": True}, {"o_scale": 0.375, "return_lse": True}):
            same(*both_ways(lambda: flash_attention_v2_cutlass(q, k, v, causal, 0.11, v_layout=v_layout, **descale, **kw)))


def test_outputs_and_status_words_of_the_caller(both_ways):
    q, k, v = tensors(2, 4, 2, 192, 192, 128, "natural")
    outs = [torch.empty(2, 4, 192, 128, dtype=torch.float16, device=DEV) for _ in range(2)]
    word = torch.zeros(1, dtype=torch.int32, device=DEV)
    left = iter(outs)
    a, b = both_ways(lambda: flash_attention_v2_cutlass(q, k, v, True, 0.1, v_layout="natural", out=next(left), _status=word))
    assert a[0].data_ptr() == outs[0].data_ptr() and b[0].data_ptr() == outs[1].data_ptr()
    same(a, b)
    # defaults: no mask, scale 1, V transposed
    vt = v.transpose(2, 3).contiguous()
    same(*both_ways(lambda: flash_attention_v2_cutlass(q, k, vt)))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(2, 3, 65, 64), (1, 2, 1, 8), (1, 5, 4096, 128)])
def test_quantisation(both_ways, shape, dtype):
    x = torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).to(dtype)
    for per_head in (False, True):
        same(*both_ways(lambda: quantize_e4m3(x, per_head=per_head)))
    y = x.reshape(-1)[:-3]
    if y.numel() > 0:
        same(*both_ways(lambda: quantize_e4m3(y)))


def test_refusals_read_the_same(both_ways, monkeypatch):
    native = api._native()
    q, k, v = tensors(1, 2, 2, 64, 64, 64, "natural")
    bad = [lambda: flash_attention_v2_cutlass(q, k, v.transpose(2, 3), False, 0.1),                              # not contiguous
           lambda: flash_attention_v2_cutlass(q, k, v, False, -1.0, v_layout="natural"),                         # scale
           lambda: flash_attention_v2_cutlass(q, k, v, False, 0.1, v_layout="natural", out=q),                   # dtype of out
           lambda: flash_attention_v2_cutlass(q, k, v, False, 0.1, v_layout="natural", descale_q=scales(3, 1)),  # length
           lambda: flash_attention_v2_cutlass(q, k, v[:, :1], False, 0.1, v_layout="natural"),
           lambda: quantize_e4m3(torch.zeros(4, 4, device=DEV)),
           lambda: quantize_e4m3(torch.zeros(4, 4, device=DEV, dtype=torch.float16), per_head=True),
           lambda: quantize_e4m3(torch.zeros(2, 2, 3, device=DEV, dtype=torch.float16), per_head=True)]
    for f in bad:
        said = []
        for module in (native, False):
            monkeypatch.setattr(api, "_native_module", module)
            with pytest.raises(RuntimeError) as e:
                f()
            said.append(str(e.value))
        assert said[0] == said[1]
