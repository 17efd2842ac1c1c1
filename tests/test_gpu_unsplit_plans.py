"""What is known of a sparse plan that splits no request: the merge kernel is left out, under torch.inference_mode() too, and
only as long as the plan is what it was."""
import copy
import contextlib

import pytest
import torch

import gpu_util as U
from oracle import decode, gen, quant, scheduler

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _kernels(names):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        yield
        torch.cuda.synchronize()
    names += [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]


def _case():
    t = gen.DecodeCase(b=21, s_q=1, s_k=600, is_varlen=True, topk=128, h_q=128)
    d = gen.make_decode_case(t)
    kq = quant.quantize_k_cache(d.blocked_k, t.dv, 128)
    ref = decode.decode_ref(d.cache_seqlens, d.block_table, d.q, quant.dequantize_k_cache(kq), t.dv, False, d.abs_indices)
    args = [x.cuda() for x in (d.q, kq, d.block_table, d.cache_seqlens)]
    return t, args, d.indices.cuda(), ref


def _run(args, idx, md, ns):
    import flashmla_windows_linux_sm120_b200 as fm
    q, kq, table, lens = args
    return fm.flash_mla_with_kvcache(q, kq, table, lens, 512, md, ns, is_fp8_kvcache=True, indices=idx)


def _split_plan(t, parts):
    """A valid plan of the same shape that does split requests: made for fewer partitions, the others left empty."""
    md, ns = scheduler.schedule_cut_ref([0] * t.b, 60, t.topk)
    assert ns[-1] > t.b
    md = md + [[t.b, 0, t.b - 1, 0, 0, 0, 0, 0]] * (parts - 60)
    return torch.tensor(md, dtype=torch.int32, device="cuda"), torch.tensor(ns, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("inference", [False, True])
def test_merge_kernel_is_left_out_until_the_plan_changes(inference):
    import flashmla_windows_linux_sm120_b200 as fm
    t, args, idx, ref = _case()
    with torch.inference_mode(inference):
        md, ns = fm.get_mla_metadata(args[3], t.h_q, 1, t.h_q, True, t.topk)
        assert int(ns[t.b]) == t.b
        _run(args, idx, md, ns)
        names = []
        with _kernels(names):
            out, lse = _run(args, idx, md, ns)
        assert [n for n in names if "mla_pair_kernel" in n] and not [n for n in names if "combine" in n], names
        U.assert_out_lse(out.cpu(), lse.cpu(), *ref)
        split_md, split_ns = _split_plan(t, md.shape[0])
        md.copy_(split_md)
        ns.copy_(split_ns)
        names = []
        with _kernels(names):
            out, lse = _run(args, idx, md, ns)
        assert [n for n in names if "combine" in n], names
        U.assert_out_lse(out.cpu(), lse.cpu(), *ref)


@pytest.mark.parametrize("inference", [False, True])
def test_a_copied_plan_is_a_plan_about_which_nothing_is_known(inference, tmp_path):
    import flashmla_windows_linux_sm120_b200 as fm
    t, args, idx, ref = _case()
    md, ns = fm.get_mla_metadata(args[3], t.h_q, 1, t.h_q, True, t.topk)
    torch.save(ns, tmp_path / "ns.pt")
    split_md, split_ns = _split_plan(t, md.shape[0])
    with torch.inference_mode(inference):
        for other in (copy.deepcopy(ns), torch.load(tmp_path / "ns.pt"), copy.copy(ns)):
            U.assert_out_lse(*[x.cpu() for x in _run(args, idx, md, other)], *ref)
            other.copy_(split_ns)
            U.assert_out_lse(*[x.cpu() for x in _run(args, idx, split_md, other)], *ref)
