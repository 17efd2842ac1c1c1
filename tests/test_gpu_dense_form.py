"""Which dense forwards take CTAs over: those with two CTAs per SM that have rows, not those whose grid is that large because one
sequence is longer than the others, and not those of long tiles at 192/128."""
import pytest
import torch

from test_gpu_unsplit_plans import _kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,h,d,causal,want", [
    ([1500, 700, 300, 100, 20], 16, 192, True, "false"), ([1000] + [30] * 6, 16, 128, False, "false"), ([256] * 20, 16, 192, True, "true"), ([256] * 9, 32, 128, True, "true"),
    ([256] * 8, 32, 128, True, "false"), ([16384] + [128] * 255, 1, 192, True, "true"), ([2048] * 8, 8, 192, False, "true"), ([4200] * 4, 8, 192, False, "false"),
    ([4200] * 4, 8, 192, True, "false"), ([4096] * 4, 8, 192, True, "true"), ([4200] * 4, 8, 128, False, "true")])
def test_form(lens, h, d, causal, want):
    import flashmla_windows_linux_sm120_b200 as fm
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines lie elsewhere with another number of SMs")
    n = sum(lens)
    q, k, v = (torch.zeros((n, h, w), dtype=torch.bfloat16, device="cuda") for w in (d, d, 128))
    cu = torch.tensor([0, *lens], device="cuda").cumsum(0).to(torch.int32)
    names = []
    with torch.no_grad():
        fm.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=causal)
        with _kernels(names):
            fm.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=causal)
    assert [n.split(">")[0].split(", ")[-1] for n in names if "dense_fwd_tc_kernel" in n] == [want]
