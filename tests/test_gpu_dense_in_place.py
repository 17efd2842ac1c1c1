"""dQ written over Q or over dO through the low-level call: the dQ kernel may start while the dK / dV kernel still runs, but not
where it would overwrite what that one reads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,over", [(192, "q"), (128, "q"), (128, "d_o"), (192, "part of q")])
def test_dq_in_place(d, over):
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    from flashmla_windows_linux_sm120_b200._cabi import lib
    g = torch.Generator(device="cuda").manual_seed(d)
    lens, h = [1500, 700, 2000, 1100], 16                # more tiles of either kernel than SMs
    total = sum(lens)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")

    def randn(*shape):
        return torch.randn(shape, device="cuda", generator=g, dtype=torch.bfloat16)

    wide = randn(total, 2 * h if over == "part of q" else h, d)
    q, k, v, d_o = wide[:, :h], randn(total, h, d), randn(total, h, 128), randn(total, h, 128)
    o = torch.empty_like(v)
    lse = torch.empty((h, total), device="cuda").t()
    args = (1, d ** -0.5, max(lens), max(lens))
    cuda_sm100.dense_prefill_fwd(torch.empty(0, device="cuda"), q, k, v, cu, cu, o, lse, *args)
    work = torch.empty(lib.fmla_dense_bwd_workspace_bytes(total, h, d), dtype=torch.uint8, device="cuda")

    def backward(q, d_o, dq):
        dk, dv = torch.empty_like(k), torch.empty_like(v)
        cuda_sm100.dense_prefill_bwd(work, d_o, q, k, v, o, lse, cu, cu, dq, dk, dv, *args)
        torch.cuda.synchronize()
        return dq, dk, dv

    expected = backward(q, d_o, torch.empty((total, h, d), device="cuda", dtype=torch.bfloat16))
    for _ in range(3):
        q2, d_o2 = wide.clone()[:, :h], d_o.clone()
        got = backward(q2, d_o2, d_o2 if over == "d_o" else q2)
        for name, a, b in zip(("dq", "dk", "dv"), got, expected):
            assert torch.equal(a, b), name
