"""Logits that keep growing along the keys: the scale a row carries has to move in many blocks (more than 2^8 each time),
which ordinary inputs never ask for after the first block.  Dense forward, and decode with few rows."""
import pytest
import torch

from oracle import decode, dense, gen
from oracle.check import check_is_allclose
from test_gpu_decode import _run_dense
from test_gpu_dense import LSE_TOL, TOL, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,causal", [(192, False), (192, True), (128, True)])
def test_dense_fwd_moving_scale(d, causal):
    g = torch.Generator().manual_seed(d)
    sq, sk, h = 300, 700, 2
    q = torch.randn(sq, h, d, generator=g).to(torch.bfloat16)
    k = (torch.randn(sk, h, d, generator=g) * torch.linspace(0.2, 6, sk).view(-1, 1, 1)).to(torch.bfloat16)
    v = torch.rand(sk, h, 128, generator=g).to(torch.bfloat16)
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32) for n in (sq, sk))
    c = dict(q=q, k=k, v=v, d_out=q, cu_q=cu_q, cu_k=cu_k, max_q=sq, max_k=sk, scale=d ** -0.5)
    out, lse, _ = _run(c, causal, False)
    r_out, r_lse = dense.dense_fwd_ref(q, k, v, cu_q, cu_k, causal, d ** -0.5)
    assert check_is_allclose("out", out, r_out, **TOL)
    assert check_is_allclose("lse", lse, r_lse, **LSE_TOL)


@pytest.mark.parametrize("h_q,s_q", [(16, 1), (16, 4), (32, 1)])
def test_few_rows_moving_scale(h_q, s_q):
    t = gen.DecodeCase(b=160, s_q=s_q, s_k=700, h_q=h_q, is_causal=s_q > 1)      # more requests than partitions: whole requests per CTA
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
