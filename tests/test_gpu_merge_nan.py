"""Rows whose logits are NaN, where a request or query token that is one piece to the caller is cut over several CTAs: the same
elements are NaN, and the same log-sum-exps, as where one CTA takes it."""
import ctypes as C

import pytest
import torch

from oracle import gen
from test_gpu_shared_rows_choice import _ctas_per_row

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(torch.isinf(a), torch.isinf(b)) and torch.equal(torch.signbit(a)[torch.isinf(a)], torch.signbit(b)[torch.isinf(b)])


@pytest.mark.parametrize("s_q,h_q", [(1, 128), (5, 128), (3, 64)])
def test_sparse_prefill(s_q, h_q):
    import flashmla_windows_linux_sm120_b200 as fm
    from flashmla_windows_linux_sm120_b200._cabi import SparsePrefillParams, check, lib
    n = C.c_size_t(0)
    check(lib.fmla_sparse_prefill_scratch_bytes(s_q, h_q, 2048, C.byref(n)))
    assert n.value > 0                                                   # tokens are cut
    q, kv, idx = (x.cuda() for x in gen.make_prefill_case(gen.PrefillCase(s_q=s_q, s_kv=900, topk=2048, h_q=h_q)))
    q[0, 3] = float("nan")
    q[s_q - 1, 7, 575] = float("inf")
    kv[5, 0, 550] = float("nan")
    idx[(idx == 5) & (torch.arange(s_q, device="cuda").view(-1, 1, 1) != 0)] = 6      # the first token alone sees row 5
    idx[0, 0, 1000] = 5
    got = fm.flash_mla_sparse_fwd(q, kv, idx, 576 ** -0.5)
    out, mx, lse = torch.empty((s_q, h_q, 512), dtype=torch.bfloat16, device="cuda"), torch.empty((s_q, h_q), device="cuda"), torch.empty((s_q, h_q), device="cuda")
    p = SparsePrefillParams(s_q=s_q, s_kv=900, h_q=h_q, h_kv=1, d_qk=576, d_v=512, topk=2048, sm_scale=576 ** -0.5, q=q.data_ptr(), q_stride_s=q.stride(0),
                            q_stride_h=576, kv=kv.data_ptr(), kv_stride_s=576, kv_stride_h=576, indices=idx.data_ptr(), indices_stride_s=2048,
                            indices_stride_h=2048, out=out.data_ptr(), max_logits=mx.data_ptr(), lse=lse.data_ptr())
    check(lib.fmla_sparse_prefill_fwd(C.byref(p), torch.cuda.current_stream().cuda_stream))      # without scratch nothing is cut
    assert torch.isnan(lse).any() and (s_q == 1 or not torch.isnan(lse).all())
    for a, b in zip(got, (out, mx, lse)):
        _same(a, b)


def test_shared_rows():
    import flashmla_windows_linux_sm120_b200 as fm
    t = gen.DecodeCase(b=7, s_q=1, s_k=2300, h_q=64)
    d = gen.make_decode_case(t)
    d.cache_seqlens.copy_(torch.tensor([2111, 1900, 2300, 1, 2050, 40, 2222]))
    d.q[3, 0, 9] = float("nan")
    d.q[5, 0, 2] = float("nan")
    d.q[6, 0, 30] = float("nan")
    lens = d.cache_seqlens.cuda()
    md, ns = fm.get_mla_metadata(lens, 64, 1)
    splits = ns.diff().tolist()
    assert splits[3] == 1 and splits[5] == 1 and splits[6] > 1
    out, lse = fm.flash_mla_with_kvcache(d.q.cuda(), d.blocked_k.cuda(), d.block_table.cuda(), lens, 512, md, ns)
    if md.shape[0] == 148:
        assert _ctas_per_row(md.tolist(), ns.tolist(), 148) > 1
    want = torch.zeros((7, 1, 64), dtype=torch.bool)
    want[3, 0, 9] = want[5, 0, 2] = want[6, 0, 30] = True
    assert torch.equal(torch.isnan(out).all(-1).cpu(), want) and torch.equal(torch.isnan(out).any(-1).cpu(), want)
    assert torch.isnan(lse[3, 9]).all() and torch.isnan(lse[5, 2]).all()             # whole requests to the caller
    assert (lse[6, 30] == float("inf")).all()                                        # one that the schedule splits
    assert torch.isfinite(lse).sum() == lse.numel() - 3
