"""Dense decode where several 64-row tiles read the same pages: odd numbers of query tokens with 64 heads, head counts that fill
one and a half tiles or three; lengths around page ends and causal borders, whole and split requests, moving scales, and a
padded output (C ABI)."""
import ctypes as C

import pytest
import torch

import gpu_util as U
from oracle import decode, gen
from test_gpu_decode import _run_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q,s_q,causal,fp16,h_kv", [(64, 3, True, False, 1), (64, 5, False, True, 1), (96, 1, False, False, 1), (100, 2, True, True, 1),
                                                      (192, 2, True, False, 1), (128, 3, True, False, 2)])
def test_several_tiles_per_page(h_q, s_q, causal, fp16, h_kv):
    t = gen.DecodeCase(b=12, s_q=s_q, s_k=64, h_q=h_q, h_kv=h_kv, is_causal=causal)
    lens = [1, 2, 3, 63, 64, 65, 66, 129, 130, 0, 1500, 5000]
    t.s_k = max(lens)
    d = gen.make_decode_case(t)
    for i, n in enumerate(lens):
        d.cache_seqlens[i] = n
        pages = (n + 63) // 64
        if n % 64:
            d.blocked_k[int(d.block_table[i, pages - 1]), n % 64:] = float("nan")      # beyond the sequence: never to be seen
        d.block_table[i, pages:] = 2147480000
    if fp16:
        d.q, d.blocked_k = d.q.to(torch.float16), d.blocked_k.to(torch.float16)
    out, lse, _, ns = _run_dense(d, t)
    assert int(ns[-1]) > t.b
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, d.blocked_k, t.dv, causal)
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q}")


def test_moving_scale():
    t = gen.DecodeCase(b=60, s_q=3, s_k=700, h_q=64, is_causal=True)                   # several requests per partition
    d = gen.make_decode_case(t)
    for i in range(t.b):
        pages = d.block_table[i, :11].long()
        d.blocked_k[pages] = (d.blocked_k[pages].float() * torch.linspace(1, 40, 11).view(-1, 1, 1, 1)).to(torch.bfloat16)
    out, lse, _, _ = _run_dense(d, t)
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, d.blocked_k, t.dv, True)
    # the rounding of P to 16 bits (2^-9 of sum p |v|) and of the output (2^-9 of it); lse: fp32 sums of logits up to 100
    bound = 2 ** -8 * float(torch.nan_to_num(d.blocked_k.float()).abs().max())
    assert float((out.float() - ref_out).abs().max()) <= bound
    assert float((lse - ref_lse).abs().max()) <= 1e-3


@pytest.mark.parametrize("h_q,s_q", [(64, 3), (100, 1)])
def test_strided_output(h_q, s_q):
    import flashmla_windows_linux_sm120_b200 as fm
    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    from test_zz_no_alloc import _params
    t = gen.DecodeCase(b=7, s_q=s_q, s_k=2500, h_q=h_q, is_causal=s_q > 1)
    d = gen.make_decode_case(t)
    for i, n in enumerate([64, 3, 65, 0, 2500, 130, 200]):
        d.cache_seqlens[i] = n
    cache = torch.nan_to_num(d.blocked_k)
    dev = dict(q=d.q.cuda(), kcache=cache.cuda(), block_table=d.block_table.cuda(), lens=d.cache_seqlens.cuda())
    md, ns = fm.get_mla_metadata(dev["lens"], s_q * h_q, 1)
    wide = torch.full((t.b, s_q + 1, h_q + 1, 520), -7.0, dtype=torch.bfloat16, device="cuda")
    lse = torch.full((t.b, h_q, s_q), float("nan"), device="cuda")
    rows = (t.b + md.shape[0]) * s_q * h_q
    p = _params(dev, t, md, ns, wide[:, :s_q, :h_q, :512], lse, torch.empty(rows, device="cuda"), torch.empty(rows * 512, device="cuda"))
    check(lib.fmla_fwd_kvcache_mla(C.byref(p), torch.cuda.current_stream().cuda_stream))
    wide = wide.cpu()
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, cache, 512, t.is_causal)
    U.assert_out_lse(wide[:, :s_q, :h_q, :512], lse.cpu(), ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q}")
    assert (wide[:, s_q:] == -7).all() and (wide[:, :, h_q:] == -7).all() and (wide[..., 512:] == -7).all()
