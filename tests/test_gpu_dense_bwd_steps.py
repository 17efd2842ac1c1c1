"""Dense backward with steps of 64 and of 128 streamed rows: sequences beside a long one take the longer steps, by themselves the
shorter ones, and their gradients are the same bit for bit, at every edge of either step and with NaN and Inf on either side."""
import pytest
import torch

from gpu_util import kernel_names

pytestmark = pytest.mark.gpu


def _grads(x, lens_q, lens_k, causal):
    """dq, dk, dv, and whether they come from steps of 64 rows."""
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    d = x["q"].shape[2]
    cu_q, cu_k = (torch.tensor([0, *n], device="cuda").cumsum(0).to(torch.int32) for n in (lens_q, lens_k))
    args = (int(causal), d ** -0.5, max(lens_q), max(lens_k))
    o, lse = torch.empty_like(x["d_o"]), torch.empty(x["q"].shape[:2][::-1], device="cuda").T
    cuda_sm100.dense_prefill_fwd(None, x["q"], x["k"], x["v"], cu_q, cu_k, o, lse, *args)
    grads = [torch.empty_like(x[n]) for n in "qkv"]
    work = torch.empty(4 * lse.numel() + 256, dtype=torch.uint8, device="cuda")
    call = lambda: cuda_sm100.dense_prefill_bwd(work, x["d_o"], x["q"], x["k"], x["v"], o, lse, cu_q, cu_k, *grads, *args)      # noqa: E731
    main = ["tc64_kernel" in n for n in kernel_names(call) if "dense_bwd_dq" in n or "dense_bwd_dkdv" in n]
    assert len(main) == 2 and main[0] == main[1]
    call()
    return grads, main[0]


@pytest.mark.parametrize("d", [192, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_same_gradients(d, causal):
    lens_q = [1, 2, 15, 16, 17, 63, 64, 65, 100, 127, 128, 129, 191, 192, 193, 256, 257, 320, 5]
    lens_k = [3, 2, 17, 16, 15, 65, 64, 63, 128, 130, 127, 129, 192, 190, 257, 256, 300, 320, 333]
    h, between, long = 3, 70, len(lens_q) * 2400
    g = torch.Generator(device="cuda").manual_seed(d)
    r = lambda n, w: torch.randn((n, h, w), device="cuda", dtype=torch.bfloat16, generator=g)       # noqa: E731
    short = dict(q=r(sum(lens_q), d), k=r(sum(lens_k), d), v=r(sum(lens_k), 128), d_o=r(sum(lens_q), 128))
    beside = {}
    for n, value in (("q", float("nan")), ("k", float("nan")), ("v", float("inf")), ("d_o", float("inf"))):
        parts = short[n].split(lens_q if n in ("q", "d_o") else lens_k)
        poison = torch.full((between, h, short[n].shape[2]), value, dtype=torch.bfloat16, device="cuda")
        beside[n] = torch.cat([t for part in parts for t in (part, poison)] + [r(long, poison.shape[2])])
    want, steps64 = _grads(short, lens_q, lens_k, causal)
    with_poison = [[x for n in lens for x in (n, between)] + [long] for lens in (lens_q, lens_k)]
    got, steps64_beside = _grads(beside, *with_poison, causal)
    assert steps64 and not steps64_beside
    for n, a, b, lens in zip("qkv", want, got, (lens_q, lens_k, lens_k)):
        pieces = b.split([x for m in lens for x in (m, between)] + [long])[0:-1:2]
        assert torch.equal(a, torch.cat(pieces)), n


@pytest.mark.parametrize("causal,mean,steps64", [(True, 1088, True), (True, 1090, False), (False, 352, True), (False, 354, False)])
def test_rule(causal, mean, steps64):
    g = torch.Generator(device="cuda").manual_seed(mean)
    x = {n: torch.randn((2 * mean, 1, w), device="cuda", dtype=torch.bfloat16, generator=g) for n, w in (("q", 128), ("k", 128), ("v", 128), ("d_o", 128))}
    assert _grads(x, [mean - 100, mean + 100], [mean + 30, mean - 30], causal)[1] == steps64
