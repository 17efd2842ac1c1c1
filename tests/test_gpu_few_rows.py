"""Dense decode with at most 64 query rows per CTA: every operand width (16, 32, 64 rows), whole query tokens sharing a
tile (heads a multiple of 8), one token per tile otherwise, head tiles above 64, partly filled tiles, and the lengths at
which a page, the ring of pages or the causal border ends."""
import pytest
import torch

import gpu_util as U
from oracle import decode, gen
from test_gpu_decode import _run_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h_q,h_kv,s_q,causal,fp16", [
    (1, 1, 1, False, False), (5, 1, 3, True, False), (8, 1, 1, False, True), (8, 1, 5, True, False), (16, 1, 4, True, False),
    (16, 1, 5, True, False), (20, 1, 2, True, True), (24, 1, 2, True, False), (32, 1, 3, True, False), (48, 2, 2, False, False),
    (48, 1, 2, True, False), (64, 1, 2, True, True), (96, 1, 2, True, False), (192, 2, 1, False, False),
])
def test_few_rows(h_q, h_kv, s_q, causal, fp16):
    t = gen.DecodeCase(b=9, s_q=s_q, s_k=64, h_q=h_q, h_kv=h_kv, is_causal=causal)
    # one long request among short ones: some are split, some CTAs walk many pages, some several requests
    lens = [1, 63, 64, 65, 130, 0, 1100, 3777, 257]
    t.s_k = max(lens)
    d = gen.make_decode_case(t)
    for i, n in enumerate(max(n, s_q) if n else 0 for n in lens):
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
    # Values below 1 (the generator's): with N(0, 1) a short sequence has outputs up to 4, where the rounding of P (2^-9 of
    # sum p |v|, up to 8e-3) and of the output (half a step, 8e-3) add up to more than the helper's bound of 1e-2.
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q}")


@pytest.mark.parametrize("h_q,s_q,fp16", [(5, 1, False), (8, 3, True), (16, 1, False), (24, 2, False), (32, 1, True), (64, 1, False),
                                          (64, 2, True), (100, 1, False)])
def test_few_rows_strided_output(h_q, s_q, fp16):
    """Rows leave in 16-byte pieces through shared memory: every tile width and fill, requests whole and split, into a padded
    output (C ABI) whose padding stays as it was."""
    import ctypes as C

    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    from test_zz_no_alloc import _params
    t = gen.DecodeCase(b=7, s_q=s_q, s_k=1, h_q=h_q, is_causal=s_q > 1)
    lens = [64, 1, 65, 0, 2500, 130, 200]
    t.s_k = max(lens)
    d = gen.make_decode_case(t)
    for i, n in enumerate(max(n, s_q) if n else 0 for n in lens):
        d.cache_seqlens[i] = n
    dtype = torch.float16 if fp16 else torch.bfloat16
    cache = torch.nan_to_num(d.blocked_k).to(dtype)
    dev = dict(q=d.q.to(dtype).cuda(), kcache=cache.cuda(), block_table=d.block_table.cuda(), lens=d.cache_seqlens.cuda())
    import flashmla_windows_linux_sm120_b200 as fm
    md, ns = fm.get_mla_metadata(dev["lens"], s_q * h_q, 1)
    assert t.b < int(ns[-1]) < 2 * t.b + md.shape[0]
    wide = torch.full((t.b, s_q + 1, h_q + 1, 520), -7.0, dtype=dtype, device="cuda")
    lse = torch.full((t.b, h_q, s_q), float("nan"), device="cuda")
    rows = (t.b + md.shape[0]) * s_q * h_q
    lse_acc, o_acc = torch.empty(rows, device="cuda"), torch.empty(rows * 512, device="cuda")
    p = _params(dev, t, md, ns, wide[:, :s_q, :h_q, :512], lse, lse_acc, o_acc)
    p.q_dtype = int(fp16)
    check(lib.fmla_fwd_kvcache_mla(C.byref(p), torch.cuda.current_stream().cuda_stream))
    wide = wide.cpu()
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q.to(dtype), cache, 512, t.is_causal)
    U.assert_out_lse(wide[:, :s_q, :h_q, :512], lse.cpu(), ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q}")
    assert (wide[:, s_q:] == -7).all() and (wide[:, :, h_q:] == -7).all() and (wide[..., 512:] == -7).all()
