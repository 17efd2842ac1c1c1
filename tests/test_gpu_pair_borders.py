"""CTA pairs that walk several requests or query tokens: requests and tokens of one block and of several, requests without any, and
parts of requests in between, so that every border follows work of every length on either stage of the rings."""
import pytest
import torch

import gpu_util as U
from oracle import decode, gen, quant
from test_gpu_decode import _run_dense, _run_sparse
from test_gpu_prefill import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q,s_q,lens", [(128, 1, [1, 64, 65, 0, 128, 200, 321]), (128, 1, [64]), (128, 2, [2, 0, 0, 130, 70]),
                                          (64, 2, [1, 66, 0, 129, 1000]), (128, 1, [3000, 64, 64, 1])])
def test_dense(h_q, s_q, lens):
    t = gen.DecodeCase(b=229, s_q=s_q, s_k=max(lens), h_q=h_q, is_causal=s_q > 1)
    d = gen.make_decode_case(t)
    for i in range(t.b):
        d.cache_seqlens[i] = lens[i % len(lens)]
    out, lse, _, _ = _run_dense(d, t)
    few = list(range(0, t.b, 3))                     # the oracle on a third of the requests
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens[few], d.block_table[few], d.q[few], d.blocked_k, t.dv, t.is_causal)
    U.assert_out_lse(out[few], lse[few], ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q} lens={lens}")


@pytest.mark.parametrize("topk", [64, 128, 192, 320])
def test_sparse_decode(topk):
    t = gen.DecodeCase(b=233, s_q=1, s_k=400, topk=topk)
    d = gen.make_decode_case(t)
    kq = quant.quantize_k_cache(d.blocked_k, t.dv, 128)
    out, lse = _run_sparse(d, t, kq)[:2]
    few = list(range(0, t.b, 3))
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens[few], d.block_table[few], d.q[few], quant.dequantize_k_cache(kq), t.dv, False, d.abs_indices[few])
    U.assert_out_lse(out[few].cpu(), lse[few].cpu(), ref_out, ref_lse, what=f"topk={topk}")


@pytest.mark.parametrize("s_q,topk", [(300, 64), (229, 128), (229, 192), (160, 320), (3000, 64)])
def test_sparse_prefill(s_q, topk):
    q, kv, idx = gen.make_prefill_case(gen.PrefillCase(s_q=s_q, s_kv=500, topk=topk))
    idx[s_q // 2] = -1
    _check(q, kv, idx, 576 ** -0.5, what=f"s_q={s_q} topk={topk}")
