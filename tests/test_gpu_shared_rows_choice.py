"""Which decode calls of at most 64 rows look for rows of the schedule to share: the others run a kernel without it."""
import re

import pytest
import torch

from gpu_util import kernel_names
from oracle import scheduler

pytestmark = pytest.mark.gpu


def _ctas_per_row(md, ns, parts):
    b = len(ns) - 1
    fits = [i for i in range(2, 7) if md[parts // i][0] >= b and i * ns[b] <= min(b + parts, 64 * b)]
    return max(fits, default=1) if ns[b] > 2 * b else 1


def _few_rows_forms(call):
    """Whether the attention kernel of each call is the form that looks for rows to share."""
    return [m.group(1) == "1" for m in (re.search(r"mla_few_rows_kernelILi\d+ELi\d+ELb[01]ELb([01])E", n) for n in kernel_names(call)) if m]


@pytest.mark.parametrize("b,h_q,s_q,topk", [(1, 16, 1, 64), (1, 64, 1, 2048), (5, 64, 2, 512), (8, 16, 1, 512), (16, 16, 1, 512), (16, 64, 1, 128), (20, 96, 1, 1024),
                                            (30, 64, 1, 2048), (40, 64, 1, 256), (49, 64, 1, 512), (60, 16, 1, 192), (148, 64, 1, 64), (160, 16, 1, 128)])
def test_sparse(b, h_q, s_q, topk):
    import flashmla_windows_linux_sm120_b200 as fm
    cache = torch.zeros((2, 64, 1, 656), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    q = torch.zeros((b, s_q, h_q, 576), dtype=torch.bfloat16, device="cuda")
    lens = torch.full((b,), 100, dtype=torch.int32, device="cuda")
    idx = torch.zeros((b, s_q, topk), dtype=torch.int32, device="cuda")
    md, ns = fm.get_mla_metadata(lens, s_q * h_q, 1, h_q, True, topk)
    k = _ctas_per_row(*scheduler.schedule_cut_ref([0] * b, md.shape[0], topk), md.shape[0])
    plan = md, ns.clone()                                # (a copy: nothing is known of it, so that unsplit plans come here too)
    table = torch.zeros((b, 2), dtype=torch.int32, device="cuda")
    forms = _few_rows_forms(lambda: fm.flash_mla_with_kvcache(q, cache, table, lens, 512, *plan, is_fp8_kvcache=True, indices=idx))
    assert forms == [k > 1], k


@pytest.mark.parametrize("b,h_q,width,want", [(4, 16, 16, True), (4, 16, 8, True), (4, 16, 7, False), (48, 16, 16, True), (49, 16, 16, False), (148, 16, 16, False)])
def test_dense(b, h_q, width, want):
    import flashmla_windows_linux_sm120_b200 as fm
    cache = torch.zeros((2, 64, 1, 576), dtype=torch.bfloat16, device="cuda")
    q = torch.zeros((b, 1, h_q, 576), dtype=torch.bfloat16, device="cuda")
    lens = torch.full((b,), width * 64, dtype=torch.int32, device="cuda")
    md, ns = fm.get_mla_metadata(lens, h_q, 1)
    if md.shape[0] != 148:
        pytest.skip("the line lies elsewhere with another number of SMs")
    table = torch.zeros((b, width), dtype=torch.int32, device="cuda")
    assert _few_rows_forms(lambda: fm.flash_mla_with_kvcache(q, cache, table, lens, 512, md, ns)) == [want]
