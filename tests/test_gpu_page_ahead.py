"""Decode of at most 64 rows over stretches around the length from which the next page is asked for in L2, with pages in one piece
and with padded rows (which are not), all in one partition."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [16, 64])
@pytest.mark.parametrize("tokens", [11 * 64, 11 * 64 + 1, 12 * 64, 13 * 64 - 5, 40 * 64 + 7])
def test_long_stretches(tokens, h):
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    g = torch.Generator(device="cuda").manual_seed(tokens + h)
    lens = [tokens, 70, tokens]
    pages = [(n + 63) // 64 for n in lens]
    order = torch.randperm(sum(pages), device="cuda", generator=g, dtype=torch.int32)
    table = torch.full((3, max(pages)), 2 ** 30, dtype=torch.int32, device="cuda")       # never read past a request's pages
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    wide = torch.randn((sum(pages), 64, 1, 640), device="cuda", dtype=torch.bfloat16, generator=g)
    q = torch.randn((3, 1, h, 576), device="cuda", dtype=torch.bfloat16, generator=g)
    cu_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    md, ns = torch.empty((1, 8), dtype=torch.int32, device="cuda"), torch.empty(4, dtype=torch.int32, device="cuda")
    check(lib.fmla_get_mla_metadata(cu_lens.data_ptr(), 3, 1, -1, md.data_ptr(), ns.data_ptr(), torch.cuda.current_stream().cuda_stream))
    results = [cuda_sm100.fwd_kvcache_mla(q, cache, 512, cu_lens, table, 576 ** -0.5, False, md, ns)
               for cache in (wide[..., :576], wide[..., :576].contiguous())]
    assert all(torch.equal(a, b) for a, b in zip(*results))
    for i, n in enumerate(lens):
        k = wide[table[i, :pages[i]].long(), :, 0, :576].reshape(-1, 576)[:n].double()
        p = torch.softmax(q[i, 0].double() @ k.T * 576 ** -0.5, dim=-1)
        out = p @ k[:, :512]
        # P and the output are rounded to bf16 (2^-9 each): two-norm below 2^-8 of the result
        assert (results[0][0][i, 0].double() - out).norm() <= 2 ** -8 * out.norm()


def _one_partition(q, cache, lens, table):
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    from flashmla_windows_linux_sm120_b200._cabi import check, lib
    cu_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    md, ns = torch.empty((1, 8), dtype=torch.int32, device="cuda"), torch.empty(len(lens) + 1, dtype=torch.int32, device="cuda")
    check(lib.fmla_get_mla_metadata(cu_lens.data_ptr(), len(lens), 1, -1, md.data_ptr(), ns.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return cuda_sm100.fwd_kvcache_mla(q, cache, 512, cu_lens, table, 576 ** -0.5, False, md, ns)


def test_pages_stored_head_by_head():
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 20 * 64 + 9
    pages = torch.randn((21, 2, 64, 576), device="cuda", dtype=torch.bfloat16, generator=g)
    q = torch.randn((1, 1, 32, 576), device="cuda", dtype=torch.bfloat16, generator=g)
    table = torch.randperm(21, device="cuda", generator=g, dtype=torch.int32).view(1, 21)
    out, lse = _one_partition(q, pages.transpose(1, 2), [n], table)[:2]              # [page][token][head]: rows of 576, heads 64 rows apart
    same = _one_partition(q, pages.transpose(1, 2).contiguous(), [n], table)
    assert torch.equal(out, same[0]) and torch.equal(lse, same[1])


@pytest.mark.parametrize("entry", [24, -1, 2 ** 30, -2 ** 31])
def test_entries_that_are_no_page(entry):
    """They read as pages of zeros, wherever in a long stretch they stand."""
    g = torch.Generator(device="cuda").manual_seed(4)
    cache = torch.randn((25, 64, 1, 576), device="cuda", dtype=torch.bfloat16, generator=g)
    cache[24] = 0
    q = torch.randn((1, 1, 16, 576), device="cuda", dtype=torch.bfloat16, generator=g)
    table = torch.randperm(24, device="cuda", generator=g, dtype=torch.int32).view(1, 24)
    table[0, [3, 13, 23]] = 24
    want = _one_partition(q, cache, [24 * 64], table)
    table[0, [3, 13, 23]] = entry
    got = _one_partition(q, cache[:24], [24 * 64], table)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
