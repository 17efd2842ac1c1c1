"""Sparse decode and sparse prefill where a CTA takes at most 64 query rows: every operand width (16, 32, 64 rows), partly
filled tiles, several head tiles, one block and more blocks than the ring holds, requests split or not, padding indices."""
import pytest
import torch

import gpu_util as U
from oracle import decode, gen, quant, sparse_prefill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q,s_q,topk,b", [(1, 1, 64, 3), (16, 2, 512, 5), (24, 1, 192, 2), (32, 1, 1024, 1), (64, 2, 704, 3), (64, 1, 64, 160),
                                            (96, 1, 320, 4)])
def test_sparse_decode_few_rows(h_q, s_q, topk, b):
    import flashmla_windows_linux_sm120_b200 as fm
    t = gen.DecodeCase(b=b, s_q=s_q, s_k=1500, is_varlen=True, topk=topk, h_q=h_q, seed=h_q + topk)
    d = gen.make_decode_case(t)
    kq = quant.quantize_k_cache(d.blocked_k, t.dv, 128)
    kd = quant.dequantize_k_cache(kq)
    lens = d.cache_seqlens.cuda()
    md, ns = fm.get_mla_metadata(lens, t.s_q * t.h_q, 1, t.h_q, True, t.topk)
    out, lse = fm.flash_mla_with_kvcache(d.q.cuda(), kq.cuda(), d.block_table.cuda(), lens, t.dv, md, ns, is_fp8_kvcache=True,
                                         indices=d.indices.cuda())
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, kd, t.dv, False, d.abs_indices)
    U.assert_out_lse(out.cpu(), lse.cpu(), ref_out, ref_lse, what=f"h_q={h_q} topk={topk}")


@pytest.mark.parametrize("h_q,s_q,s_kv,topk", [(64, 1, 70, 64), (64, 150, 333, 192), (192, 3, 200, 128), (64, 5, 2000, 1024)])
def test_sparse_prefill_few_rows(h_q, s_q, s_kv, topk):
    import flashmla_windows_linux_sm120_b200 as fm
    g = torch.Generator().manual_seed(s_q)
    q = (torch.randn(s_q, h_q, 576, generator=g) / 2).to(torch.bfloat16)
    kv = (torch.randn(s_kv, 1, 576, generator=g) / 2).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(max(s_kv, topk), generator=g)[:topk] for _ in range(s_q)]).to(torch.int32).unsqueeze(1)
    idx[idx >= s_kv] = -1
    idx[:, :, ::13] = s_kv + 5                        # out of range: padding
    if s_q > 2:
        idx[1] = -1                                   # a token without any key
    out, mx, lse = (x.cpu() for x in fm.flash_mla_sparse_fwd(q.cuda(), kv.cuda(), idx.cuda(), 576 ** -0.5))
    r_out, r_mx, r_lse = sparse_prefill.sparse_prefill_ref(q, kv, idx, 576 ** -0.5, 512)
    ok = torch.isfinite(r_lse)
    assert torch.equal(torch.isfinite(lse), ok) and torch.equal(torch.isfinite(mx), torch.isfinite(r_mx))
    U.assert_target_bounds(out, lse[ok], r_out, r_lse[ok], what=f"s_q={s_q}")
    assert float((mx[ok] - r_mx[ok]).abs().max()) <= 1e-4 * 1.4427
