"""Which dense forwards take CTAs over: those with two CTAs per SM that have rows, not those whose grid is that large because one
sequence is longer than the others, and not those of long tiles at 192/128."""
import pytest
import torch

from gpu_util import kernel_names

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,h,d,causal,want", [
    ([1500, 700, 300, 100, 20], 16, 192, True, False), ([1000] + [30] * 6, 16, 128, False, False), ([256] * 20, 16, 192, True, True), ([256] * 9, 32, 128, True, True),
    ([256] * 8, 32, 128, True, False), ([16384] + [128] * 255, 1, 192, True, True), ([2048] * 8, 8, 192, False, True), ([4200] * 4, 8, 192, False, False),
    ([4200] * 4, 8, 192, True, False), ([4096] * 4, 8, 192, True, True), ([4200] * 4, 8, 128, False, True)])
def test_form(lens, h, d, causal, want):
    import flashmla_windows_linux_sm120_b200 as fm
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines lie elsewhere with another number of SMs")
    n = sum(lens)
    q, k, v = (torch.zeros((n, h, w), dtype=torch.bfloat16, device="cuda") for w in (d, d, 128))
    cu = torch.tensor([0, *lens], device="cuda").cumsum(0).to(torch.int32)
    with torch.no_grad():
        names = kernel_names(lambda: fm.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=causal))
    assert [f"dense_fwd_tc_kernelILi{d}ELb{int(want)}E" in n for n in names if "dense_fwd_tc_kernel" in n] == [True], names
