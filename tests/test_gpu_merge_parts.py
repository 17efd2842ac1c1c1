"""The merge of split requests around the lines of its launch rule: warps per row and parts in flight by the number of rows, fewer
parts than are asked for at once, more than a warp has lanes, and partial slots that nobody wrote; and that it ends behind the
attention kernel, whether or not it finds anything to merge."""
import os
import re

import pytest
import torch

import gpu_util as U
from oracle import decode, gen, quant
from test_gpu_decode import _run_dense, _run_sparse

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_windows_linux_sm120_b200", "csrc")


def test_the_schedule_is_complete_when_the_merge_starts():
    """The merge of a decode reads the schedule before it waits for the attention kernel.  That holds because each CTA of each
    attention kernel waits for the kernels in front of it before it lets the merge start."""
    for name in ("mla_pair.cu", "mla_few_rows.cu", "mla_tile64.cu"):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        assert text.count("pdl_allow_dependents();") == 1 and text.count("pdl_wait();") == 1, name
        between = text[text.index("pdl_wait();"):text.index("pdl_allow_dependents();")]
        assert between.split() == ["pdl_wait();"], name
        start = text[text.rindex("__global__", 0, text.index("pdl_wait();")):text.index("pdl_wait();")]
        assert "return;" not in start, name


def test_the_merge_ends_behind_the_attention_kernel():
    """What follows a decode in a stream, or in a graph, is ordered behind the merge alone.  So no thread of a merge kernel leaves
    before the wait for the kernel in front: where nothing is split, the whole grid would."""
    with open(os.path.join(CSRC, "combine.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for kernel in ("decode_combine_kernel(const", "sparse_prefill_combine_kernel(const"):
        body = text[text.index(kernel):]
        body = body[:body.index("\n}\n")]
        assert body.count("pdl_wait();") == 1, kernel
        ahead = body[:body.index("pdl_wait();")]
        assert "return" not in re.sub(r"const auto \w+ = \[&\] \{.*?\n  \};", "", ahead, flags=re.S), kernel
        line = ahead[ahead.rindex("\n"):]
        assert line == "\n  ", f"{kernel}: the wait stands under a condition"


def _poison():
    """What the allocator hands out next holds NaN: an unwritten partial that reached a sum would show."""
    torch.cuda.empty_cache()
    del_me = [torch.full((1 << 22,), float("nan"), device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    del del_me


@pytest.mark.gpu
@pytest.mark.parametrize("h_q,lens", [
    (16, [1024, 900, 0, 1]), (64, [2111, 65, 1500, 64]), (64, [1200, 1, 640, 1300, 0]), (64, [2111, 1900, 2300, 1, 2050, 0, 2222]),
    (64, [900] * 9 + [0]), (64, [500, 1, 0, 700] * 4), (64, [9000]), (16, [3000] * 37), (16, [130, 9000, 0, 64] * 9), (128, [700, 0, 9000, 1])])
def test_dense(h_q, lens):
    t = gen.DecodeCase(b=len(lens), s_q=1, s_k=max(lens), h_q=h_q)
    d = gen.make_decode_case(t)
    d.cache_seqlens.copy_(torch.tensor(lens))
    for i, n in enumerate(lens):
        if n % 64:
            d.blocked_k[int(d.block_table[i, n // 64]), n % 64:] = float("nan")
    _poison()
    out, lse, _, _ = _run_dense(d, t)
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, d.blocked_k, t.dv, False)
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"h_q={h_q} lens={lens[:7]}")


@pytest.mark.gpu
@pytest.mark.parametrize("h_q,s_q,b", [(64, 1, 1), (64, 1, 4), (64, 2, 3), (64, 2, 5), (128, 1, 6)])
def test_sparse(h_q, s_q, b):
    t = gen.DecodeCase(b=b, s_q=s_q, s_k=1500, is_varlen=True, topk=512, h_q=h_q, seed=b)
    d = gen.make_decode_case(t)
    d.indices[0] = -1                                       # every part of the first request is empty
    d.abs_indices[0] = -1
    kq = quant.quantize_k_cache(d.blocked_k, t.dv, 128)
    _poison()
    out, lse = _run_sparse(d, t, kq)
    ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, quant.dequantize_k_cache(kq), t.dv, False, d.abs_indices)
    U.assert_out_lse(out, lse, ref_out, ref_lse, what=f"h_q={h_q} s_q={s_q} b={b}")


@pytest.mark.gpu
@pytest.mark.parametrize("h_q,s_q,lens", [(16, 1, [2048] * 128), (16, 1, [40] * 300), (64, 1, [64] * 90), (64, 3, [50] * 60), (128, 1, [2048] * 64)])
def test_what_follows_an_unsplit_decode_sees_its_outputs(h_q, s_q, lens):
    """One decode whose schedule splits no request, and readers of its outputs right behind it in the same graph."""
    import flashmla_windows_linux_sm120_b200 as fm
    b, pages = len(lens), (max(lens) + 63) // 64
    gen_ = torch.Generator(device="cuda").manual_seed(b)
    cache = torch.randn((b * pages, 64, 1, 576), generator=gen_, device="cuda", dtype=torch.bfloat16)
    table = torch.randperm(b * pages, generator=gen_, device="cuda", dtype=torch.int32).view(b, pages)
    qs = [torch.randn((b, s_q, h_q, 576), generator=gen_, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    n = torch.tensor(lens, dtype=torch.int32, device="cuda")
    plan = fm.get_mla_metadata(n, s_q * h_q, 1)
    assert (plan[1].diff() == 1).all()                      # nothing to merge
    q = qs[0].clone()

    def decode():
        return fm.flash_mla_with_kvcache(q, cache, table, n, 512, *plan)

    expected = []
    for x in qs:
        q.copy_(x)
        expected.append([y.clone() for y in decode()])
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, lse = decode()
        copied = out.clone(), lse.clone()                   # copy nodes
        negated = -out, -lse                                # kernels
    for r in range(20):
        q.copy_(qs[r % 2])
        for y in (out, lse, *copied, *negated):
            y.fill_(float("nan"))
        graph.replay()
        for want, a, c in zip(expected[r % 2], copied, negated):
            assert torch.equal(a, want) and torch.equal(-c, want), r
