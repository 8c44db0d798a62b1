"""Few query rows against many keys (no causal mask, V as [keys, head_dim]): the decode kernel, and
the folding of query heads that share a key/value head into one slice.

Against a model of it (the same rounding of P to fp8, starting maximum over the first 64 keys) the
difference is the order of fp32 sums and, now and then, a P on the other side of a rounding step: 2e-3 as
for the prefill kernel.  Against the fp32 oracle it is the rounding of P: 3e-2 (e5m2 6e-2)."""
import ctypes
import math

import pytest
import torch

from cutlass_flash_atten_fp8_b200 import _lib, check_status, flash_attention_v2_cutlass
from oracle.attention_oracle import error_metrics

pytestmark = pytest.mark.gpu


def rand8(*shape, seed, dtype=torch.float8_e4m3fn, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def call(q, k, v, scale, **kw):
    d = torch.device("cuda", 0)
    n = q.numel()
    guard = torch.full((n + 64,), float("nan"), dtype=torch.float16, device=d)
    out, lse = flash_attention_v2_cutlass(q.to(d), k.to(d), v.to(d), False, scale, v_layout="natural", return_lse=True,
                                          out=guard[:n].view(q.shape), **kw)
    check_status(d)
    assert bool(torch.isnan(guard[n:]).all())
    return out.float().cpu(), lse.cpu()


def reference(q, k, v, scale):
    g = q.shape[1] // k.shape[1]
    s = q.float() @ k.float().repeat_interleave(g, 1).transpose(2, 3) * scale
    return torch.softmax(s, -1) @ v.float().repeat_interleave(g, 1), torch.logsumexp(s, -1)


def rounded_p(q, k, v, scale, dtype):
    """P relative to the maximum over the first 64 keys, rounded to fp8 for P V but not for the row sum."""
    g = q.shape[1] // k.shape[1]
    s = q.float() @ k.float().repeat_interleave(g, 1).transpose(2, 3) * scale
    p = torch.exp(s - s[..., :64].amax(-1, keepdim=True))
    assert float(p.max()) <= 448.0                  # the maximum is not raised
    return p.to(dtype).float() @ v.float().repeat_interleave(g, 1) / p.sum(-1, keepdim=True)


def taken(slices, rows, Sk, D):
    """Whether the call goes to the decode kernel (fa8::decode_takes)."""
    f = _lib.load()._ZN3fa812decode_takesElliii
    f.restype, f.argtypes = ctypes.c_bool, [ctypes.c_int64, ctypes.c_int64] + 3 * [ctypes.c_int]
    return f(slices, rows, Sk, D, torch.cuda.get_device_properties(0).multi_processor_count)


# one key, less than the first 64, not a multiple of a 32-key step, one step more than a split of two to
# eight CTAs of four warps; 1, 2, 7, 8, 9, 16 and 17 rows; 64 and 65 (past the decode kernel: folded prefill)
@pytest.mark.parametrize("H,Hk,Sq,Sk,D", [
    (2, 2, 1, 1, 32), (2, 1, 1, 33, 64), (4, 2, 1, 64, 128), (7, 1, 1, 65, 128), (8, 1, 1, 1000, 256), (3, 1, 3, 777, 96),
    (2, 1, 8, 4097, 64), (17, 1, 1, 2049, 160), (16, 2, 8, 1056, 128), (5, 1, 13, 513, 192), (8, 1, 2, 288, 224)])
@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
def test_against_the_oracles(H, Hk, Sq, Sk, D, dtype):
    q, k, v = (rand8(2, h, s, D, seed=Sk + i, dtype=dtype) for i, (h, s) in enumerate([(H, Sq), (Hk, Sk), (Hk, Sk)]))
    scale = 1 / math.sqrt(D)
    e4m3 = dtype == torch.float8_e4m3fn
    out, lse = call(q, k, v, scale)
    assert error_metrics(out, rounded_p(q, k, v, scale, dtype))["rel_l2"] <= 2e-3
    ref, ref_lse = reference(q, k, v, scale)
    assert float((lse - ref_lse).abs().max()) <= 1e-5 * float(ref_lse.abs().max()) + 1e-5
    # scores of a few units: the maximum over the first 64 keys is outgrown by later ones
    q6 = (q.float() * 6).to(dtype)
    out, lse = call(q6, k, v, scale)
    ref, ref_lse = reference(q6, k, v, scale)
    assert error_metrics(out, ref)["rel_l2"] <= (3e-2 if e4m3 else 6e-2)
    assert float((lse - ref_lse).abs().max()) <= 1e-5 * float(ref_lse.abs().max()) + 1e-5


@pytest.mark.parametrize("Sq,Sk", [(1, 700), (3, 700), (100, 300)])
def test_scales_per_head_follow_the_heads_of_a_group(Sq, Sk):
    H, Hk, D = 6, 2, 64
    q, k, v = rand8(2, H, Sq, D, seed=1), rand8(2, Hk, Sk, D, seed=2), rand8(2, Hk, Sk, D, seed=3)
    d = torch.device("cuda", 0)
    dq, dk, dv = (0.5 + torch.rand(2 * n, generator=torch.Generator().manual_seed(n)) for n in (H, Hk, Hk))
    out, lse = call(q, k, v, 0.125, descale_q=dq.to(d), descale_k=dk.to(d), descale_v=dv.to(d))
    ref, ref_lse = reference(q.float() * dq.view(2, H, 1, 1), k.float() * dk.view(2, Hk, 1, 1), v.float() * dv.view(2, Hk, 1, 1), 0.125)
    assert error_metrics(out, ref)["rel_l2"] <= 3e-2
    assert float((lse - ref_lse).abs().max()) <= 1e-4


def test_a_stale_status_word_leaves_the_output_alone():
    d = torch.device("cuda", 0)
    q, k, v = (rand8(1, 2, s, 64, seed=s).to(d) for s in (1, 512, 512))
    word = torch.ones(1, dtype=torch.int32, device=d)
    out = torch.full((1, 2, 1, 64), 7.0, dtype=torch.float16, device=d)
    flash_attention_v2_cutlass(q, k, v, False, 0.125, v_layout="natural", out=out, _status=word)
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())
    with pytest.raises(RuntimeError):              # the host has been told; the next call reports it
        flash_attention_v2_cutlass(q, k, v, False, 0.125, v_layout="natural", out=out, _status=word)
    word.zero_()
    flash_attention_v2_cutlass(q, k, v, False, 0.125, v_layout="natural", out=out, _status=word)
    check_status(d, word=word)
    assert not bool((out == 7.0).any())


@pytest.mark.parametrize("D,col", [(32, 5), (64, 63), (96, 40), (128, 0), (192, 150), (256, 255)])
@pytest.mark.parametrize("Sk", [1, 33, 70, 999])
def test_an_infinite_value_of_the_last_key_comes_through(D, col, Sk):
    # keys past the last one take no part: 0 * inf there would be a NaN
    q, k, v = (rand8(1, 1, s, D, seed=s, dtype=torch.float8_e5m2) for s in (1, Sk, Sk))
    plain, _ = call(q, k, v, 0.01)
    v[0, 0, Sk - 1, col] = float("inf")
    out, _ = call(q, k, v, 0.01)
    assert float(out[0, 0, 0, col]) == math.inf
    plain[0, 0, 0, col] = math.inf
    assert torch.equal(out, plain)


# blocks of rows: one more row than fits a block, the last block full or of one row, at either end of the kernels'
# head dims; the most rows there are, and one more.  A row's output is rounded to fp16 (2^-11) after sums in another
# order: 1e-3.  The kernel's fp32 exponentials are off by about 3e-7 of their value and roundings lie 2^-4 to 2^-3 of it
# apart (e5m2 2^-3 to 2^-2), so of the 1e5 to 3e5 probabilities of a case one or two may be rounded the other way: such a row
# is off by a step of its largest P (at most 2^-3, e5m2 2^-2, of it) times that key's value.
@pytest.mark.parametrize("rows,group", [(17, 17), (32, 4), (33, 3), (48, 6), (63, 7)])
@pytest.mark.parametrize("D", [32, 64, 96, 128, 160, 256])
def test_several_row_blocks(rows, group, D):
    Hk, Sk = (1, 1500) if D % 64 else (2, 2049)
    assert taken(2 * Hk, rows, Sk, D) and not taken(2 * Hk, 64, Sk, D)
    dtype = torch.float8_e5m2 if rows == 33 else torch.float8_e4m3fn
    q, k, v = (rand8(2, h, s, D, seed=Sk + i, dtype=dtype) for i, (h, s) in enumerate([(group * Hk, rows // group), (Hk, Sk), (Hk, Sk)]))
    scale = 1 / math.sqrt(D)
    out, lse = call(q, k, v, scale)
    want = rounded_p(q, k, v, scale, dtype)
    ref, ref_lse = reference(q, k, v, scale)
    off, size = (out - want).norm(dim=-1), want.norm(dim=-1)
    # P relative to the row sum: exp(largest score - log-sum-exp)
    s = q.float() @ k.float().repeat_interleave(group, 1).transpose(2, 3) * scale
    step = (0.25 if rows == 33 else 0.125) * torch.exp(s.amax(-1) - ref_lse) * v.float().norm(dim=-1).max()
    turned = off > 1e-3 * size
    assert int(turned.sum()) <= 2
    assert bool((off <= 1e-3 * size + 2 * step * turned).all())
    assert float((lse - ref_lse).abs().max()) <= 1e-5 * float(ref_lse.abs().max()) + 1e-5


@pytest.mark.parametrize("rows,Sk", [(18, 2000), (63, 1300), (195, 300), (390, 500)])
def test_scales_per_head_over_row_blocks_and_folded_tiles(rows, Sk):
    Sq = rows // 3                                   # groups of three heads: heads share a block of rows or a tile
    assert taken(4, rows, Sk, 64) == (rows < 64)
    assert rows < 64 or (rows + 127) // 128 < 3 * ((Sq + 127) // 128)          # folded
    test_scales_per_head_follow_the_heads_of_a_group(Sq, Sk)
