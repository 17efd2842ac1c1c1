"""What the native marshalling of the dense calls accepts and refuses."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _args(d=192, h=2, n=70):
    g = torch.Generator(device="cuda").manual_seed(d)
    r = lambda *shape: torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=g)       # noqa: E731
    cu = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    return dict(q=r(n, h, d), k=r(n, h, d), v=r(n, h, 128), cu_q=cu, cu_k=cu, o=torch.empty((n, h, 128), device="cuda", dtype=torch.bfloat16),
                lse=torch.empty((h, n), device="cuda").T, code=1, scale=d ** -0.5, max_q=n, max_k=n)


def _fwd(a):
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    cuda_sm100.dense_prefill_fwd(None, *(a[n] for n in ("q", "k", "v", "cu_q", "cu_k", "o", "lse", "code", "scale", "max_q", "max_k")))
    return a["o"].clone(), a["lse"].clone()


def test_numbers_of_any_kind():
    a = _args()
    want = _fwd(a)
    for same in (dict(max_q=np.int64(70), max_k=torch.tensor(70)), dict(max_q=70.0, scale=np.float64(a["scale"])), dict(code=True), dict(code=1.0)):
        assert all(torch.equal(x, y) for x, y in zip(_fwd(dict(a, **same)), want)), same
    for other in (0, 2, None):                           # anything but 1: no mask
        assert not torch.equal(_fwd(dict(a, code=other))[0], want[0])


@pytest.mark.parametrize("change,message", [(dict(q="cpu"), "q must be on CUDA"), (dict(k="float"), "must be bfloat16"), (dict(lse="bf16"), "lse must be float32"),
                                            (dict(cu_q="long"), "cumulative seqlens must be int32"), (dict(v="2-D"), "bad ranks"),
                                            (dict(q="strided"), "last dimensions must be contiguous"), (dict(k="short"), "k shape mismatch"),
                                            (dict(o="short"), "o shape mismatch"), (dict(lse="short"), "lse must be"), (dict(scale=0.0), "softmax_scale")])
def test_what_is_refused(change, message):
    a = _args()
    how = {"cpu": lambda t: t.cpu(), "float": lambda t: t.float(), "bf16": lambda t: t.to(torch.bfloat16), "long": lambda t: t.long(), "2-D": lambda t: t[:, 0],
           "strided": lambda t: torch.empty((70, 2, 384), device="cuda", dtype=torch.bfloat16)[:, :, ::2], "short": lambda t: t[:-1]}
    (name, what), = change.items()
    a[name] = how[what](a[name]) if isinstance(what, str) else what
    with pytest.raises(RuntimeError, match=message):
        _fwd(a)


def test_backward_refuses():
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    a = _args()
    _fwd(a)
    fixed = [a[n] for n in ("q", "k", "v")], [a[n] for n in ("o", "lse", "cu_q", "cu_k")], [a[n] for n in ("code", "scale", "max_q", "max_k")]

    def bwd(work=torch.empty(70 * 2 * 4 + 256, dtype=torch.uint8, device="cuda"), d_o=torch.zeros_like(a["o"]), dq=None):
        grads = [torch.empty_like(t) for t in fixed[0]]
        cuda_sm100.dense_prefill_bwd(work, d_o, *fixed[0], *fixed[1], grads[0] if dq is None else dq, *grads[1:], *fixed[2])
        return grads

    assert all((g == 0).all() for g in bwd())
    with pytest.raises(RuntimeError, match="workspace_buffer too small: need 768 bytes"):
        bwd(work=torch.empty(700, dtype=torch.uint8, device="cuda"))
    with pytest.raises(RuntimeError, match="gradient shape mismatch"):
        bwd(dq=torch.empty((69, 2, 192), dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(RuntimeError, match="must be bfloat16"):
        bwd(d_o=torch.zeros((70, 2, 128), device="cuda"))


def test_short_cumulative_lengths():
    """The kernels read batch + 1 entries of both (more keys' entries than that are never looked at)."""
    a = _args()
    want = _fwd(a)
    with pytest.raises(RuntimeError, match="cumulative_seqlen_kv is shorter"):
        _fwd(dict(a, cu_k=a["cu_k"][:1]))
    with pytest.raises(RuntimeError, match="cumulative_seqlen_kv is shorter"):
        _fwd(dict(a, cu_q=torch.tensor([0, 30, 70], dtype=torch.int32, device="cuda")))
    longer = torch.tensor([0, 70, 10 ** 6], dtype=torch.int32, device="cuda")
    assert all(torch.equal(x, y) for x, y in zip(_fwd(dict(a, cu_k=longer)), want))
