"""Dense decode with 64 heads and an even number of query tokens: a CTA pair holds two consecutive tokens, which read the same
pages and see different borders."""
import pytest
import torch

import gpu_util as U
from oracle import decode, gen
from test_gpu_decode import _run_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s_q,causal,fp16,h_kv", [(2, True, False, 1), (2, False, True, 1), (4, True, True, 1), (6, True, False, 1),
                                                  (2, True, False, 2)])
def test_two_tokens_per_pair(s_q, causal, fp16, h_kv):
    t = gen.DecodeCase(b=12, s_q=s_q, s_k=64, h_q=64 * h_kv, h_kv=h_kv, is_causal=causal)
    # the two borders in one page, on either side of a page's end (65: token 0 sees 64 keys), tokens without any key
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
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"s_q={s_q} h_kv={h_kv}")


@pytest.mark.parametrize("s_q", [2, 4])
def test_two_tokens_per_pair_moving_scale(s_q):
    t = gen.DecodeCase(b=90, s_q=s_q, s_k=700, h_q=64, is_causal=True)                 # whole requests and several per pair
    d = gen.make_decode_case(t)
    for i in range(t.b):
        pages = d.block_table[i, :11].long()
        d.blocked_k[pages] = (d.blocked_k[pages].float() * torch.linspace(1, 40, 11).view(-1, 1, 1, 1)).to(torch.bfloat16)
    out, lse, _, _ = _run_dense(d, t)
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, d.blocked_k, t.dv, t.is_causal)
    # the rounding of P to 16 bits (2^-9 of sum p |v|) and of the output (2^-9 of it); lse: fp32 sums of logits up to 100
    bound = 2 ** -8 * float(torch.nan_to_num(d.blocked_k.float()).abs().max())
    assert float((out.float() - ref_out).abs().max()) <= bound
    assert float((lse - ref_lse).abs().max()) <= 1e-3
