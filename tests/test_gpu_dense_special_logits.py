"""Dense forward with logits that ordinary inputs do not make: a row with a NaN or an infinite logit comes out as NaN, wherever the key
stands among those that the two ways of forming 2^x take in turn, and the other rows are as without it; logits far below the row's
largest give exactly nothing."""
import pytest
import torch

from oracle import dense
from oracle.check import check_is_allclose
from test_gpu_dense import LSE_TOL, TOL, _run

pytestmark = pytest.mark.gpu
NAN, INF = float("nan"), float("inf")


def _case(d, sq, sk, seed):
    g = torch.Generator().manual_seed(seed)
    q, k = (torch.randn(n, 1, d, generator=g).to(torch.bfloat16) for n in (sq, sk))
    v = torch.rand(sk, 1, 128, generator=g).to(torch.bfloat16)
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32) for n in (sq, sk))
    return dict(q=q, k=k, v=v, d_out=q, cu_q=cu_q, cu_k=cu_k, max_q=sq, max_k=sk, scale=d ** -0.5)


@pytest.mark.parametrize("d", [192, 128])
@pytest.mark.parametrize("key", [0, 1, 2, 3, 4, 5, 6, 31, 63, 64, 100, 127, 130, 299])
@pytest.mark.parametrize("bad", [NAN, INF])
def test_nan_and_infinite_logits(bad, key, d):
    c = _case(d, 200, 300, key)
    c["q"][:, 0, 0] = 1.0                                    # every row sees the sign of what the key holds here
    c["k"][key, 0, 0] = bad
    c["q"][7, 0, 0] = c["q"][150, 0, 0] = -1.0               # rows for which an infinite key is minus infinity: it takes no part
    out, lse, _ = _run(c, False, False)
    keeps = torch.zeros(200, dtype=torch.bool)
    if bad == INF:
        keeps[[7, 150]] = True
    assert torch.isnan(out[~keeps]).all() and torch.isnan(lse[~keeps]).all()
    if keeps.any():
        rest = torch.arange(300) != key
        ref, ref_lse = dense.dense_fwd_ref(c["q"][keeps], c["k"][rest], c["v"][rest], torch.tensor([0, 2]), torch.tensor([0, 299]), False, c["scale"])
        assert check_is_allclose("out", out[keeps], ref, **TOL) and check_is_allclose("lse", lse[keeps], ref_lse, **LSE_TOL)


@pytest.mark.parametrize("d", [192, 128])
def test_a_nan_row_leaves_the_others(d):
    c = _case(d, 300, 300, d)
    clean, clean_lse, _ = _run(c, True, False)
    c["q"][[5, 129, 290]] = NAN
    out, lse, _ = _run(c, True, False)
    bad = torch.isnan(c["q"].float()).any(-1).any(-1)
    assert torch.isnan(out[bad]).all() and torch.isnan(lse[bad]).all()
    assert torch.equal(out[~bad], clean[~bad]) and torch.equal(lse[~bad], clean_lse[~bad])


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("spread", [30.0, 120.0, 128.0, 3000.0])
def test_far_below_the_largest(spread, causal):
    """Logits (base 2) between 0 and -spread along the keys, in shuffled order, so that many lie around and below the smallest normal
    number; values up to 1."""
    d, sq, sk = 128, 140, 400
    c = _case(d, sq, sk, int(spread))
    c["q"].zero_()
    c["k"].zero_()
    c["q"][:, 0, 0] = 1.0
    order = torch.randperm(sk, generator=torch.Generator().manual_seed(1))
    c["k"][:, 0, 0] = (-spread * order / sk * 0.6931471805599453 / c["scale"]).to(torch.bfloat16)
    out, lse, _ = _run(c, causal, False)
    ref, ref_lse = dense.dense_fwd_ref(c["q"], c["k"], c["v"], c["cu_q"], c["cu_k"], causal, c["scale"])
    assert check_is_allclose("out", out, ref, **TOL) and check_is_allclose("lse", lse, ref_lse, **LSE_TOL)


@pytest.mark.parametrize("n", [100, 500])                    # steps of 64 and of 128 streamed rows
@pytest.mark.parametrize("row", [0, 1, 2, 3, 4, 5, 30, 33, 62, 99])
def test_a_nan_row_reaches_its_gradients(row, n):
    """The log-sum-exp of the row is NaN, so its P is, whichever way it is formed: dQ of the row, dK and dV of every key it sees."""
    c = _case(128, n, n, n + row)
    c["d_out"] = torch.randn(n, 1, 128, generator=torch.Generator().manual_seed(row)).to(torch.bfloat16)
    c["q"][row] = NAN
    _, _, (dq, dk, dv) = _run(c, True, True)
    assert torch.isnan(dq[row]).all() and torch.isnan(dk[:row + 1]).all() and torch.isnan(dv[:row + 1]).all()
    rest = torch.arange(n) != row
    assert not torch.isnan(dq[rest]).any() and not torch.isnan(dv[row + 1:]).any()      # (dK of other keys: zero times the row itself)
