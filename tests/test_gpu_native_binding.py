"""What the native marshalling of the per-step calls owes its caller besides results: other threads and error types."""
import threading
import time

import pytest
import torch

from oracle import gen

pytestmark = pytest.mark.gpu


def test_a_full_launch_queue_stops_no_other_thread():
    """A launch waits while the stream's queue is full; the GIL must be free meanwhile."""
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    kv = torch.randn(1, 576, device="cuda", dtype=torch.bfloat16)
    cache = torch.zeros((1, 64, 1, 656), dtype=torch.float8_e4m3fn, device="cuda")
    slots = torch.zeros(1, dtype=torch.int32, device="cuda")
    cuda_sm100.quantize_kv_fp8(kv, cache, slots)
    torch.cuda.synchronize()
    gaps, done = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    ticker = threading.Thread(target=tick)
    ticker.start()
    torch.cuda._sleep(900_000_000)                       # about half a second, then the queue below runs off
    start = time.perf_counter()
    for _ in range(3000):
        cuda_sm100.quantize_kv_fp8(kv, cache, slots)
    waited = time.perf_counter() - start
    done.set()
    ticker.join()
    torch.cuda.synchronize()
    assert waited > 0.3, "the launch queue never filled"
    assert max(gaps) < 0.25, max(gaps)


def test_two_threads_decode_on_their_own_streams():
    import flashmla_windows_linux_sm120_b200 as fm
    from test_gpu_decode import _run_dense
    cases = [gen.DecodeCase(b=3, s_q=1, s_k=900, h_q=16, is_varlen=True, seed=1), gen.DecodeCase(b=9, s_q=2, s_k=400, h_q=128, is_varlen=True, is_causal=True, seed=2)]
    data = [gen.make_decode_case(t) for t in cases]
    expected = [_run_dense(d, t)[:2] for d, t in zip(data, cases)]
    on_gpu = [[x.cuda() for x in (d.q, d.blocked_k, d.block_table, d.cache_seqlens)] for d in data]
    torch.cuda.synchronize()
    results, errors = [[], []], []

    def work(k):
        try:
            t, (q, cache, table, lens) = cases[k], on_gpu[k]
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(50):
                    md, ns = fm.get_mla_metadata(lens, t.s_q * t.h_q, 1)
                    results[k].append(fm.flash_mla_with_kvcache(q, cache, table, lens, 512, md, ns, causal=t.is_causal))
                torch.cuda.current_stream().synchronize()
        except Exception as e:                            # noqa: BLE001  shown below, in the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not errors, errors
    for k in range(2):
        for out, lse in results[k]:
            assert torch.equal(out.cpu(), expected[k][0]) and torch.equal(lse.cpu(), expected[k][1])


def test_errors_keep_their_types():
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    one = dict(dtype=torch.bfloat16, device="cuda")
    n = 1 << 23                                          # an output of half a terabyte: refused before anything is launched
    q, kv = torch.zeros((1, 64, 576), **one).expand(n, 64, 576), torch.zeros((1, 1, 576), **one)
    idx = torch.zeros((1, 1, 64), dtype=torch.int32, device="cuda").expand(n, 1, 64)
    with pytest.raises(torch.OutOfMemoryError):
        cuda_sm100.sparse_prefill_fwd(q, kv, idx, 1.0)
    with pytest.raises(IndexError):                      # a tensor without dimensions, where the batch is asked for
        cuda_sm100.get_mla_decoding_metadata(torch.tensor(5, dtype=torch.int32, device="cuda"), 128, 1)
    lens = torch.tensor([64], dtype=torch.int32, device="cuda")
    with pytest.raises(TypeError):
        cuda_sm100.get_mla_decoding_metadata(lens, None, 1)
    with pytest.raises(RuntimeError, match="seqlens_k must have dtype int32"):
        cuda_sm100.get_mla_decoding_metadata(lens.long(), 128, 1)
    md, ns = cuda_sm100.get_mla_decoding_metadata(lens, 128, 1)
    q, cache, table = torch.zeros((1, 1, 128, 576), **one), torch.zeros((1, 64, 1, 576), **one), torch.zeros((1, 1), dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="head_size_v == 512"):
        cuda_sm100.fwd_kvcache_mla(q, cache, 256, lens, table, 1.0, False, md, ns)
