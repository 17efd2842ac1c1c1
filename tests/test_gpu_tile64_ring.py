"""The rings of the 64-row tile kernel (five stages of half a block, which Q passes through too, and three of the last columns) over
several query tokens or requests per CTA: one block and few, odd and even, so that a token starts at every stage of the rings."""
import math

import pytest
import torch

import gpu_util as U
from oracle import decode, gen
from test_gpu_decode import _run_dense
from test_gpu_prefill import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q,s_q,topk", [(64, 700, 64), (64, 449, 128), (64, 445, 192), (64, 330, 320), (64, 297, 448), (192, 150, 192)])
def test_prefill(h_q, s_q, topk):
    q, kv, idx = gen.make_prefill_case(gen.PrefillCase(s_q=s_q, s_kv=800, topk=topk, h_q=h_q))
    idx[s_q // 2] = -1                                                                # a token without a valid index between others
    idx[3::7, :, -64:] = -1
    _check(q, kv, idx, 1 / math.sqrt(576), what=f"h_q={h_q} s_q={s_q} topk={topk}")


@pytest.mark.parametrize("h_q,s_q,blocks", [(64, 3, [1, 0, 2, 3]), (64, 3, [5, 1, 1, 0, 4]), (96, 1, [1, 2, 0, 7]), (192, 1, [3, 3, 1])])
def test_dense(h_q, s_q, blocks):
    lens = [max(64 * n - 17 * (i % 3), 0) for i, n in enumerate(blocks * (200 // len(blocks)))]
    t = gen.DecodeCase(b=len(lens), s_q=s_q, s_k=max(lens), h_q=h_q, is_causal=s_q > 1)
    d = gen.make_decode_case(t)
    d.cache_seqlens.copy_(torch.tensor(lens))
    for i, n in enumerate(lens):
        if n % 64:
            d.blocked_k[int(d.block_table[i, n // 64]), n % 64:] = float("nan")      # beyond the sequence: never to be seen
    out, lse, _, _ = _run_dense(d, t)
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, d.blocked_k, t.dv, t.is_causal)
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q} blocks={blocks}")
