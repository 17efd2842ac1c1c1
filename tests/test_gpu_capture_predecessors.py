"""Dependent launches captured into a CUDA graph behind whatever a program may have put in front of them: nothing, a fill, a
copy, a join of two streams.  Replays with other inputs against eager calls."""
import pytest
import torch

from oracle import gen, quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("front", ["nothing", "fill", "copy", "join", "event"])
@pytest.mark.parametrize("h_q,sparse", [(16, False), (128, False), (64, True), (128, True)])
def test_decode_captured_behind(front, h_q, sparse):
    import flashmla_windows_linux_sm120_b200 as fm
    t = gen.DecodeCase(b=6, s_q=1, s_k=900, h_q=h_q, is_varlen=True, topk=192 if sparse else None)
    d = gen.make_decode_case(t)
    cache = (quant.quantize_k_cache(d.blocked_k, 512, 128) if sparse else torch.nan_to_num(d.blocked_k)).cuda()
    table, lens = d.block_table.cuda(), d.cache_seqlens.cuda()
    qs = [d.q.cuda(), torch.randn_like(d.q).cuda()]
    idx = d.indices.cuda() if sparse else None
    plan = fm.get_mla_metadata(lens, h_q, 1, h_q, True, 192) if sparse else fm.get_mla_metadata(lens, h_q, 1)
    q, source, junk = qs[0].clone(), qs[0].clone(), torch.empty(1 << 20, device="cuda")

    def decode():
        return fm.flash_mla_with_kvcache(q, cache, table, lens, 512, *plan, is_fp8_kvcache=sparse, indices=idx)

    expected = []
    for x in qs:
        q.copy_(x)
        expected.append([y.clone() for y in decode()])
    q.copy_(qs[0])
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        here = torch.cuda.current_stream()
        if front == "fill":
            junk.zero_()
        elif front == "copy":
            q.copy_(source)
        elif front in ("join", "event"):
            side.wait_stream(here)
            with torch.cuda.stream(side):
                q.copy_(source)
            if front == "join":
                junk.add_(1)
            here.wait_stream(side)
        out = decode()
        again = decode()                                  # behind the merge kernel, or behind the attention kernel itself
    for n, x in ((0, qs[0]), (1, qs[1]), (0, qs[0])):
        (source if front in ("copy", "join", "event") else q).copy_(x)
        graph.replay()
        for got in (out, again):
            assert torch.equal(got[0], expected[n][0]) and torch.equal(got[1], expected[n][1])


def test_dense_backward_captured():
    import flashmla_windows_linux_sm120_b200 as fm
    lens = [300, 700]
    cu = torch.tensor([0, 300, 1000], dtype=torch.int32, device="cuda")
    q, k, v, g = (torch.randn(1000, 8, w, device="cuda", dtype=torch.bfloat16) for w in (192, 192, 128, 128))
    q, k, v = (x.requires_grad_() for x in (q, k, v))

    def step():
        out, _ = fm.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=True)
        return torch.autograd.grad(out, (q, k, v), g)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        expected = step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        grads = step()
    for _ in range(3):
        for x in grads:
            x.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(grads, expected))
