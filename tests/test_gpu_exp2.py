"""2^x as the dense kernels form part of it, on the multiply-add pipe (f2_exp2 and f2_exp2_to_128 in csrc/fmla_common.cuh): the function by
itself against 64 bits, and what its ends come to in the forward and in the backward."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest
import torch

from flashmla_windows_linux_sm120_b200 import build

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")

KERNEL = """
#include "fmla_common.cuh"
template <bool kTo128>
__global__ void each(const float* x, float* y, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  const fmla::F2 v = {x[2 * i], x[2 * i + 1]}, r = kTo128 ? fmla::f2_exp2_to_128(v) : fmla::f2_exp2(v);
  y[2 * i] = r.lo;
  y[2 * i + 1] = r.hi;
}
extern "C" int run(const float* x, float* y, int pairs, int to_128, void* stream) {
  const auto s = static_cast<cudaStream_t>(stream);
  if (to_128) each<true><<<(pairs + 255) / 256, 256, 0, s>>>(x, y, pairs);
  else each<false><<<(pairs + 255) / 256, 256, 0, s>>>(x, y, pairs);
  return static_cast<int>(cudaGetLastError());
}
"""


@pytest.fixture(scope="module")
def exp2(tmp_path_factory):
    folder = tmp_path_factory.mktemp("exp2")
    source, library = folder / "each.cu", folder / "each.so"
    source.write_text(KERNEL)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-I", build.CSRC, "-I", build.INCLUDE_DIR, "-o", str(library), str(source)], check=True)
    lib = ctypes.CDLL(str(library))
    lib.run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]

    def call(x, to_128):
        assert x.numel() % 2 == 0
        d = x.cuda()
        y = torch.empty_like(d)
        assert lib.run(d.data_ptr(), y.data_ptr(), d.numel() // 2, to_128, torch.cuda.current_stream().cuda_stream) == 0
        return y.cpu()

    return call


@pytest.mark.parametrize("to_128", [0, 1])
def test_against_64_bits(exp2, to_128):
    # 2^22 arguments over the range and as many around 0, where most of a row's lie
    x = torch.cat([torch.linspace(-126, 127.99, 1 << 22), torch.linspace(-8, 8, 1 << 22)])
    y = exp2(x, to_128).numpy().astype(np.float64)
    rel = np.abs(y / np.exp2(x.numpy().astype(np.float64)) - 1)
    print(f"[exp2] largest relative error {rel.max():.3e}")
    # the polynomial's 1.08e-7 and one rounding, 2^-24; the roundings before it are scaled by |f q(f)| < 0.42 and its derivative
    assert rel.max() <= 1.08e-7 + 2.0 ** -24 + 0.1 * 2.0 ** -24
    below = torch.linspace(-127, -126, 1 << 12)
    assert np.abs(exp2(below, to_128).numpy().astype(np.float64) - np.exp2(below.numpy().astype(np.float64))).max() <= 2.0 ** -127      # less than the smallest normal number


@pytest.mark.parametrize("to_128", [0, 1])
def test_the_ends(exp2, to_128):
    big = [128.0] if to_128 else [128.0, 128.3, 129.0, 200.0, 255.0, 256.0, 300.0, 383.0, 384.0, 512.0, 1e4, 1e6, 4.2e6, 1.3e7, 1e9, 3e38, INF]
    assert (exp2(torch.tensor(big + [128.0]), to_128) == INF).all()
    assert (exp2(torch.tensor([-127.0, -127.5, -128.0, -150.0, -256.0, -512.0, -1e4, -1e6, -1.3e7, -1e9, -3e38, -INF]), to_128) == 0).all()
    got = exp2(torch.tensor([NAN, 1.0, 2.0, NAN]), to_128)
    assert got[1] == 2 and got[2] == 4
    assert (got[[0, 3]] == 0).all() if to_128 else torch.isnan(got[[0, 3]]).all()


def test_backward_with_a_log_sum_exp_far_too_small():
    """The log-sum-exp comes from the caller: where a logit exceeds it by 2^7 and more (base 2), P is infinite, at every key."""
    from flashmla_windows_linux_sm120_b200 import cuda_sm100
    for n in (100, 500):                                     # steps of 64 and of 128 streamed rows
        q, k = (torch.zeros((n, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        v = torch.zeros_like(q)
        o, do = torch.zeros_like(q), torch.zeros_like(q)
        cu = torch.tensor([0, n], dtype=torch.int32, device="cuda")
        work = torch.empty(4 * n + 4096, dtype=torch.uint8, device="cuda")
        for excess in (129.0, 200.0, 256.5, 300.0, 1000.0):
            lse = torch.full((1, n), 0.0, device="cuda").T
            lse[5] = -excess * math.log(2)
            do.zero_()
            do[5] = 1
            dq, dk, dv = (torch.empty_like(q) for _ in range(3))
            cuda_sm100.dense_prefill_bwd(work, do, q, k, v, o, lse, cu, cu, dq, dk, dv, 0, 1.0, n, n)
            assert (dv == INF).all(), (n, excess)


def _forward(q, k, v, scale):
    import flashmla_windows_linux_sm120_b200 as fm
    cu = torch.tensor([0, q.shape[0]], dtype=torch.int32, device="cuda")
    return fm.flash_attn_varlen_func(q, k, v, cu, cu, q.shape[0], q.shape[0], softmax_scale=scale, causal=False)


@pytest.mark.parametrize("n", [12, 250])
def test_forward_where_the_scaled_logit_is_rounded_by_more_than_the_range(n):
    """Row i sees key i alone, with a logit of 2^34 and more (base 2).  Its scaled value is rounded to a multiple of 2048, and the row's largest
    exponent is what the rounding took away.  Above 2^7 the row overflows, which has to show whichever key holds it; below, it vanishes."""
    scale, seen = np.float32(1.4426950408889634), [0, 0]
    row = torch.arange(n)
    for m in range(129, 256, 1 if n < 100 else 9):
        s = np.float32(m * 2.0 ** 27)                        # two bf16 values, their product exact in fp32
        left = float(s) * float(scale) - float(np.float32(s * scale))
        if abs(left) < 160:
            continue
        q, k = (torch.zeros((n, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        # two rows share a direction, and are told apart by a second one with the sign against the other's keys
        q[row, 0, row % 125], k[row, 0, row % 125] = 2.0 ** 17, m * 2.0 ** 10
        for a in range(2):
            q[row[row // 125 != a], 0, 125 + a] = -2.0 ** 20
            k[row[row // 125 == a], 0, 125 + a] = m * 2.0 ** 10
        out, lse = _forward(q, k, torch.ones_like(q), 1.0)
        seen[left > 0] += 1
        if left > 0:
            assert torch.isnan(out).all() and not lse.isfinite().any(), (m, left)
        else:
            assert (out == 0).all() and (lse == -INF).all(), (m, left)
    assert min(seen) > 2
