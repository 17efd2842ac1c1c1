"""The kernels of a decode step are programmatic dependents of one another: a kernel is resident, waiting, while the one in
front of it still writes the schedule or the partials it will read.  Plan and decode run back to back here, without a
synchronisation or a copy between them, in buffers that are used again by plans of very different lengths."""
import os
import re

import pytest
import torch

import gpu_util as U
from oracle import decode, gen, quant

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashmla_windows_linux_sm120_b200", "csrc")


def test_no_invariant_loads_of_what_the_kernel_in_front_writes():
    """__ldg may be moved above the wait for that kernel, and is undefined for memory written while this one is resident."""
    def source(name):
        with open(os.path.join(CSRC, name)) as f:
            return re.sub(r"//[^\n]*", "", f.read())

    combine = source("combine.cu")
    merge = combine[combine.index("combine_weights(int"):combine.index("combine_partials_kernel(")]
    for name, text in [(n, source(n)) for n in ("mla_work.cuh", "mla_pair.cu", "mla_few_rows.cu")] + [("combine.cu", merge)]:
        # the FP8 records alone: their addresses come from plain loads after the wait
        assert all("rec" in arg for arg in re.findall(r"__ldg\(([^;]*);", text)), name


def test_an_empty_schedule_row_asks_for_no_work():
    """begin_idx of an empty row is the batch size: reading that request's length or split count is out of range.  Such a CTA
    has to stay (it waits for the kernel in front), so both decode kernels leave every role out instead."""
    for name, guard in (("mla_pair.cu", "if (misaligned || tile.n_work == 0) {"), ("mla_few_rows.cu", "if (n_work == 0 || misaligned) {")):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        kernel = text[text.index("pdl_wait();"):]
        assert guard in kernel
        assert not re.search(r"get_work<|request\(0\)", kernel[:kernel.index(guard)])


def _lengths(kind):
    return {"even": [700] * 12, "one_long": [70] * 11 + [6400], "other_long": [3000] + [1] * 10 + [0]}[kind]


@pytest.mark.gpu
@pytest.mark.parametrize("h_q,s_q", [(16, 1), (16, 3), (64, 1), (128, 1), (128, 2)])
def test_plan_and_decode_back_to_back_dense(h_q, s_q):
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    kinds = ["even", "one_long", "other_long"]
    sets = []
    for kind in kinds:
        t = gen.DecodeCase(b=12, s_q=s_q, s_k=6400, h_q=h_q, is_causal=s_q > 1)
        d = gen.make_decode_case(t)
        for i, n in enumerate(_lengths(kind)):
            d.cache_seqlens[i] = max(n, s_q) if n else 0
        sets.append((t, d))
    t, d = sets[0]                                          # one cache, three vectors of lengths
    q, cache, table = d.q.cuda(), torch.nan_to_num(d.blocked_k).cuda(), d.block_table.cuda()
    lens = [x.cache_seqlens.cuda() for _, x in sets]
    parts = cuda_sm100.get_mla_decoding_metadata(lens[0], s_q * h_q, 1)[0].shape[0]
    md = torch.empty((parts, 8), dtype=torch.int32, device="cuda")
    ns = torch.empty((t.b + 1,), dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    outs = []
    torch.cuda.synchronize()
    for r in range(30):
        n = lens[r % 3]
        check(lib.fmla_get_mla_metadata(n.data_ptr(), t.b, parts, -1, md.data_ptr(), ns.data_ptr(), stream))
        outs.append(cuda_sm100.fwd_kvcache_mla(q, cache, 512, n, table, 576 ** -0.5, t.is_causal, md, ns))
    torch.cuda.synchronize()
    for r in range(3, 30):
        assert torch.equal(outs[r][0], outs[r % 3][0]) and torch.equal(outs[r][1], outs[r % 3][1]), (r, kinds[r % 3])
    for k in range(3):
        ref_out, ref_lse = decode.decode_ref(sets[k][1].cache_seqlens, d.block_table, d.q, cache.cpu(), 512, t.is_causal)
        U.assert_out_lse(outs[k][0].cpu(), outs[k][1].cpu(), ref_out, ref_lse, what=f"h_q={h_q} {kinds[k]}")


@pytest.mark.gpu
@pytest.mark.parametrize("h_q", [16, 64, 128])
def test_plan_and_decode_back_to_back_sparse(h_q):
    """Plans with 320 and with 64 keys a request, made into the same buffers; most partitions of the second are empty."""
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    t = gen.DecodeCase(b=5, s_q=1, s_k=1500, is_varlen=True, topk=320, h_q=h_q)
    d = gen.make_decode_case(t)
    kq = quant.quantize_k_cache(d.blocked_k, 512, 128)
    kd = quant.dequantize_k_cache(kq)
    q, cache, table, lens = d.q.cuda(), kq.cuda(), d.block_table.cuda(), d.cache_seqlens.cuda()
    idx = [d.indices.cuda(), d.indices[:, :, 128:192].contiguous().cuda()]
    parts = cuda_sm100.get_mla_decoding_metadata(lens, h_q, 1, h_q, True, 320)[0].shape[0]
    md = torch.empty((parts, 8), dtype=torch.int32, device="cuda")
    ns = torch.empty((t.b + 1,), dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    outs = []
    torch.cuda.synchronize()
    for r in range(20):
        i = idx[r % 2]
        check(lib.fmla_get_mla_metadata(lens.data_ptr(), t.b, parts, i.shape[2], md.data_ptr(), ns.data_ptr(), stream))
        outs.append(cuda_sm100.fwd_kvcache_mla(q, cache, 512, lens, table, 576 ** -0.5, False, md, ns, True, i))
    torch.cuda.synchronize()
    for r in range(2, 20):
        assert torch.equal(outs[r][0], outs[r % 2][0]) and torch.equal(outs[r][1], outs[r % 2][1]), r
    for k, a in enumerate((d.abs_indices, d.abs_indices[:, :, 128:192])):
        ref_out, ref_lse = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, kd, 512, False, a)
        U.assert_out_lse(outs[k][0].cpu(), outs[k][1].cpu(), ref_out, ref_lse, what=f"h_q={h_q} topk={320 if k == 0 else 64}")
