"""What the speed of this package is measured on: the attention calls that a serving or training program makes.

Every case is one pass through the public entry points with inputs, cache and (for decode) the split-KV plan already
on the GPU.  Values are N(0, 1) in the stored type, the distribution of the benchmark; pages, slots and top-k positions
are shuffled.  Sequence lengths depend on the case alone, so that its work is known; everything else follows the seed.
"""
import math
import random

import torch

import flashmla_windows_linux_sm120_b200 as fm
from flashmla_windows_linux_sm120_b200 import cuda_sm100

D, DV, PAGE = 576, 512, 64
DEV = "cuda"


def listed():
    return [
        # The smallest decode step: four short requests, 16 heads (a tensor-parallel shard), plan and attention in one
        # go.  Latency, launches and host work are what a user waits for here.
        dict(name="decode_b4_h16_1k_with_plan", kind="decode", b=4, s_q=1, h_q=16, mean_len=1024, ragged=False,
             causal=False, dtype="bf16", plan=True),
        # A layer of a decode step of a full server: 128 requests around 4 k tokens, all 128 heads.
        dict(name="decode_b128_h128_4k", kind="decode", b=128, s_q=1, h_q=128, mean_len=4096, ragged=True, causal=True,
             dtype="bf16", plan=False),
        # The same with one speculated token per request: two causal query tokens.
        dict(name="decode_b128_h128_4k_sq2", kind="decode", b=128, s_q=2, h_q=128, mean_len=4096, ragged=True,
             causal=True, dtype="bf16", plan=False),
        # A tensor-parallel shard of 16 heads over a mid-size batch of longer contexts: the cache is the work.
        dict(name="decode_b61_h16_6k", kind="decode", b=61, s_q=1, h_q=16, mean_len=6000, ragged=True, causal=False,
             dtype="bf16", plan=False),
        # 64 heads, float16 cache, a handful of requests of odd lengths.
        dict(name="decode_b7_h64_2k_fp16", kind="decode", b=7, s_q=1, h_q=64, mean_len=2111, ragged=True, causal=False,
             dtype="fp16", plan=False),
        # Sparse attention decode over the FP8 cache: 64 requests of 32 k tokens, the 2048 best of each.
        dict(name="sparse_decode_b64_h128_top2048", kind="sparse_decode", b=64, s_q=1, h_q=128, topk=2048,
             seqlen=32768, plan=False),
        # The same for few requests with two query tokens each, 64 heads; the plan is made in the call.
        dict(name="sparse_decode_b5_h64_sq2_top512", kind="sparse_decode", b=5, s_q=2, h_q=64, topk=512, seqlen=9000,
             plan=True),
        # Sparse prefill of a 4096-token chunk at the end of a 32 k context.
        dict(name="sparse_prefill_4096_h128_top2048", kind="sparse_prefill", s_q=4096, h_q=128, s_kv=32768, topk=2048),
        # A short ragged chunk of a prompt, 64 heads.
        dict(name="sparse_prefill_333_h64_top512", kind="sparse_prefill", s_q=333, h_q=64, s_kv=5003, topk=512),
        # Dense causal prefill with 128-wide heads and grouped keys, a few prompts of odd lengths (inference only).
        dict(name="mha_fwd_d128_gqa_3seq", kind="mha", nseq=3, lo=700, hi=2500, h_q=32, h_k=8, d_qk=128, causal=True,
             backward=False),
        # A training step of the dense path: 8 sequences of 1 k to 8 k tokens, 128 heads of 192 / 128, causal.
        dict(name="mha_train_8seq_h128", kind="mha", nseq=8, lo=1024, hi=8192, h_q=128, h_k=128, d_qk=192, causal=True,
             backward=True),
        # The cache writer: a prefill chunk quantised into scattered slots of the FP8 cache.
        dict(name="cache_write_8192", kind="cache_write", tokens=8192, slots=65536),
    ]


def _log_int(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "sparse_decode", "sparse_decode", "sparse_prefill",
                       "sparse_prefill", "mha", "mha", "mha", "cache_write"])
    if kind == "decode":
        b = _log_int(rng, 1, 128)
        return dict(kind=kind, b=b, s_q=rng.choice([1, 1, 1, 2, 3]), h_q=rng.choice([16, 32, 64, 128, 128]),
                    mean_len=_log_int(rng, 200, min(32768, 600000 // b)), ragged=rng.random() < 0.8,
                    causal=rng.random() < 0.5, dtype=rng.choice(["bf16", "bf16", "fp16"]), plan=rng.random() < 0.3)
    if kind == "sparse_decode":
        return dict(kind=kind, b=_log_int(rng, 1, 64), s_q=rng.choice([1, 1, 2]), h_q=rng.choice([64, 128, 128]),
                    topk=64 * _log_int(rng, 2, 32), seqlen=_log_int(rng, 2100, 32768), plan=rng.random() < 0.3)
    if kind == "sparse_prefill":
        s_q = _log_int(rng, 1, 4096)
        return dict(kind=kind, s_q=s_q, h_q=rng.choice([64, 128, 128]), s_kv=s_q + _log_int(rng, 100, 28672),
                    topk=64 * _log_int(rng, 2, 32))
    if kind == "mha":
        h_q, d_qk = rng.choice([(8, 128), (32, 128), (16, 192), (128, 192)])
        backward = rng.random() < 0.5
        h_k = h_q if backward or rng.random() < 0.5 else max(1, h_q // 4)
        lo = _log_int(rng, 60, 2048)
        return dict(kind=kind, nseq=rng.randint(1, 8), lo=lo, hi=min(4096, lo * rng.randint(1, 4)), h_q=h_q, h_k=h_k,
                    d_qk=d_qk, causal=rng.random() < 0.7, backward=backward)
    tokens = _log_int(rng, 1, 60000)
    return dict(kind=kind, tokens=tokens, slots=65536)


def _lens(case):
    """Sequence lengths of a decode or dense case: a function of the case alone."""
    if case["kind"] == "mha":
        # one from each of nseq equal stretches of [lo, hi], in shuffled order
        n, lo, width = case["nseq"], case["lo"], case["hi"] - case["lo"]
        rng = random.Random("%d %d %d" % (n, lo, width))
        lens = [lo + int(width * (i + rng.random()) / n) for i in range(n)]
        rng.shuffle(lens)
        return lens
    if not case["ragged"]:
        return [case["mean_len"]] * case["b"]
    m = case["mean_len"]
    rng = random.Random("%d %d" % (case["b"], m))
    return [max(case["s_q"], rng.randint(m - m // 4, m + m // 4)) for _ in range(case["b"])]


def _positions(rows, hi, topk, gen):
    """[rows, topk] distinct positions below hi (a [rows] tensor), one from each of topk equal stretches, in shuffled
    order; rows with hi < topk take every position and are padded with -1."""
    j = torch.arange(topk, device=DEV, dtype=torch.float64)
    u = torch.rand((rows, topk), device=DEV, generator=gen, dtype=torch.float64) * 0.999
    n = torch.minimum(hi, torch.full_like(hi, topk)).unsqueeze(1)
    edge = torch.floor(j * hi.unsqueeze(1).double() / n)
    width = torch.floor((j + 1) * hi.unsqueeze(1).double() / n) - edge
    pos = (edge + torch.floor(u * width)).long()
    pos[j.unsqueeze(0) >= n] = -1
    order = torch.rand((rows, topk), device=DEV, generator=gen).argsort(dim=1)
    return torch.gather(pos, 1, order)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    cpu = torch.Generator().manual_seed(seed)

    def randn(*shape, dtype=torch.bfloat16):
        return torch.randn(shape, device=DEV, dtype=dtype, generator=gen)

    kind = case["kind"]
    st = dict(case=case)
    if kind == "decode":
        dtype = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
        lens = _lens(case)
        pages = [(n + PAGE - 1) // PAGE for n in lens]
        perm = torch.randperm(sum(pages), generator=cpu).to(torch.int32)
        table = torch.zeros((len(lens), max(pages)), dtype=torch.int32)
        at = 0
        for i, n in enumerate(pages):
            table[i, :n] = perm[at:at + n]
            at += n
        st.update(q=randn(case["b"], case["s_q"], case["h_q"], D, dtype=dtype),
                  cache=randn(sum(pages), PAGE, 1, D, dtype=dtype), table=table.to(DEV),
                  lens=torch.tensor(lens, dtype=torch.int32, device=DEV))
        if not case["plan"]:
            st["plan"] = fm.get_mla_metadata(st["lens"], case["s_q"] * case["h_q"], 1)
    elif kind == "sparse_decode":
        b, s_q, topk, seqlen = case["b"], case["s_q"], case["topk"], case["seqlen"]
        per = (seqlen + PAGE - 1) // PAGE
        table = torch.randperm(b * per, generator=cpu).to(torch.int32).view(b, per).to(DEV)
        cache = torch.empty((b * per, PAGE, 1, 656), dtype=torch.float8_e4m3fn, device=DEV)
        for p0 in range(0, b * per, 4096):
            cache[p0:p0 + 4096] = cuda_sm100.quantize_kv_fp8(randn(min(4096, b * per - p0), PAGE, 1, D))
        hi = torch.full((b * s_q,), seqlen, dtype=torch.int64, device=DEV)
        pos = _positions(b * s_q, hi, topk, gen).view(b, s_q * topk)
        slots = torch.gather(table.long(), 1, pos.clamp(min=0) // PAGE) * PAGE + pos % PAGE
        slots[pos < 0] = -1
        slots[:, ::97] = -1                                   # some padding slots, as a top-k kernel leaves them
        st.update(q=randn(b, s_q, case["h_q"], D), cache=cache, table=table,
                  lens=torch.full((b,), seqlen, dtype=torch.int32, device=DEV),
                  indices=slots.to(torch.int32).view(b, s_q, topk))
        if not case["plan"]:
            st["plan"] = fm.get_mla_metadata(st["lens"], s_q * case["h_q"], 1, case["h_q"], True, topk)
    elif kind == "sparse_prefill":
        s_q, s_kv = case["s_q"], case["s_kv"]
        # query t is the (s_kv - s_q + t)-th token of its context and sees no later one
        hi = (torch.arange(s_q, device=DEV) + (s_kv - s_q + 1)).clamp(min=1)
        st.update(q=randn(s_q, case["h_q"], D), kv=randn(s_kv, 1, D),
                  indices=_positions(s_q, hi, case["topk"], gen).to(torch.int32).view(s_q, 1, case["topk"]))
    elif kind == "mha":
        lens = _lens(case)
        total = sum(lens)
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        grad = case["backward"]
        st.update(q=randn(total, case["h_q"], case["d_qk"]).requires_grad_(grad),
                  k=randn(total, case["h_k"], case["d_qk"]).requires_grad_(grad),
                  v=randn(total, case["h_k"], 128).requires_grad_(grad),
                  cu=torch.tensor(cu, dtype=torch.int32, device=DEV), longest=max(lens))
        if grad:
            st["d_out"] = randn(total, case["h_q"], 128)
    else:
        st.update(kv=randn(case["tokens"], D),
                  cache=torch.zeros((case["slots"] // PAGE, PAGE, 1, 656), dtype=torch.float8_e4m3fn, device=DEV),
                  slots=torch.randperm(case["slots"], generator=cpu)[:case["tokens"]].to(torch.int32).to(DEV))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("decode", "sparse_decode"):
        sparse = kind == "sparse_decode"
        if case["plan"]:
            extra = (case["h_q"], True, case["topk"]) if sparse else ()
            plan = fm.get_mla_metadata(st["lens"], case["s_q"] * case["h_q"], 1, *extra)
        else:
            plan = st["plan"]
        return fm.flash_mla_with_kvcache(st["q"], st["cache"], st["table"], st["lens"], DV, *plan,
                                         causal=not sparse and case["causal"], is_fp8_kvcache=sparse,
                                         indices=st.get("indices"))
    if kind == "sparse_prefill":
        return fm.flash_mla_sparse_fwd(st["q"], st["kv"], st["indices"], D ** -0.5)
    if kind == "mha":
        q, k, v = st["q"], st["k"], st["v"]
        args = (q, k, v, st["cu"], st["cu"], st["longest"], st["longest"])
        if not case["backward"]:
            with torch.no_grad():
                return fm.flash_attn_varlen_func(*args, causal=case["causal"])
        q.grad = k.grad = v.grad = None
        out, lse = fm.flash_attn_varlen_func(*args, causal=case["causal"])
        out.backward(st["d_out"])
        return out.detach(), lse, q.grad, k.grad, v.grad
    return cuda_sm100.quantize_kv_fp8(st["kv"], st["cache"], st["slots"]).view(torch.uint8)


def work(case):
    kind = case["kind"]
    if kind == "decode":
        lens, s_q, h = _lens(case), case["s_q"], case["h_q"]
        seen = sum(lens) * s_q
        if case["causal"]:
            seen -= len(lens) * s_q * (s_q - 1) // 2
        rows = len(lens) * s_q * h
        return dict(bytes=sum(lens) * D * 2 + rows * (D * 2 + DV * 2 + 4) + sum(4 * ((n + 63) // 64) for n in lens),
                    flops=2 * h * (D + DV) * seen)
    if kind == "sparse_decode":
        rows, keys = case["b"] * case["s_q"] * case["h_q"], case["b"] * case["s_q"] * case["topk"]
        return dict(bytes=keys * (656 + 4) + rows * (D * 2 + DV * 2 + 4), flops=2 * case["h_q"] * (D + DV) * keys)
    if kind == "sparse_prefill":
        s_q, topk, h = case["s_q"], case["topk"], case["h_q"]
        keys = sum(min(topk, max(1, case["s_kv"] - s_q + 1 + t)) for t in range(s_q))
        return dict(bytes=case["s_kv"] * D * 2 + s_q * topk * 4 + s_q * h * (D * 2 + DV * 2 + 8),
                    flops=2 * h * (D + DV) * keys)
    if kind == "mha":
        lens, h, hk, d = _lens(case), case["h_q"], case["h_k"], case["d_qk"]
        pairs = sum(n * (n + 1) // 2 if case["causal"] else n * n for n in lens)
        total = sum(lens)
        nbytes = 2 * total * (h * (d + 128) + hk * (d + 128)) + 4 * total * h
        flops = 2 * h * pairs * (d + 128)
        if case["backward"]:
            nbytes += 2 * total * (h * 128 + h * d + hk * (d + 128))
            flops += 2 * h * pairs * (3 * d + 2 * 128)
        return dict(bytes=nbytes, flops=flops)
    return dict(bytes=case["tokens"] * (D * 2 + 656 + 4), flops=case["tokens"] * DV * 3)


def tolerance(case):
    # About four times the errors of the outputs against the same mathematics in 64 bits on these inputs.  Two-norm:
    # 1.8e-3 to 2.2e-3 for bf16 outputs (their own rounding and that of P), 2.5e-4 for float16, 2.4e-3 for gradients.
    # Largest difference: 2e-2 (the first rows of a causal sequence), 8e-4 for float16, 4e-2 for gradients.
    if case["kind"] == "cache_write":
        return "exact"
    if case.get("dtype") == "fp16":
        return {"rel": 1e-3, "max": 4e-3}
    return {"rel": 1e-2, "max": 0.16} if case.get("backward") else {"rel": 8.5e-3, "max": 0.08}


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits and plain torch."""
    kind = case["kind"]
    if kind == "cache_write":
        return None                          # bytes, compared bit for bit
    st = prepare(case, seed)
    with torch.no_grad():
        return dict(decode=_exact_decode, sparse_decode=_exact_sparse_decode, sparse_prefill=_exact_sparse_prefill,
                    mha=_exact_mha)[kind](st)


def _attend(q, k, v, scale, visible=None):
    """softmax(scale q k^T) v over the visible keys, its natural log-sum-exp and its largest scaled logit."""
    s = (q @ k.transpose(-1, -2)) * scale
    if visible is not None:
        s.masked_fill_(~visible, -math.inf)
    lse = torch.logsumexp(s, dim=-1)
    top = s.amax(dim=-1)
    return torch.exp_(s.sub_(lse.unsqueeze(-1))) @ v, lse, top


def _exact_decode(st):
    case = st["case"]
    b, s_q, h = case["b"], case["s_q"], case["h_q"]
    out = torch.empty((b, s_q, h, DV), dtype=torch.float64, device=DEV)
    lse = torch.empty((b, h, s_q), dtype=torch.float64, device=DEV)
    for i, n in enumerate(st["lens"].tolist()):
        k = st["cache"][st["table"][i, :(n + PAGE - 1) // PAGE].long()].reshape(-1, D)[:n].double()
        for t in range(s_q):
            seen = n - (s_q - 1 - t) if case["causal"] else n
            out[i, t], lse[i, :, t], _ = _attend(st["q"][i, t].double(), k[:seen], k[:seen, :DV], D ** -0.5)
    return out, lse


def _exact_sparse_decode(st):
    case = st["case"]
    b, s_q, h = case["b"], case["s_q"], case["h_q"]
    records = st["cache"].view(torch.uint8).view(-1, 656)
    out = torch.empty((b, s_q, h, DV), dtype=torch.float64, device=DEV)
    lse = torch.empty((b, h, s_q), dtype=torch.float64, device=DEV)
    for i in range(b):
        slots = st["indices"][i].long()
        rec = records[slots.clamp(min=0)]                                          # [s_q, topk, 656]
        nope = rec[..., :DV].contiguous().view(torch.float8_e4m3fn).float().unflatten(-1, (4, 128))
        nope = (nope * rec[..., 512:528].contiguous().view(torch.float32).unsqueeze(-1)).to(torch.bfloat16).flatten(-2)
        k = torch.cat([nope, rec[..., 528:].contiguous().view(torch.bfloat16)], dim=-1).double()
        out[i], l, _ = _attend(st["q"][i].double(), k, k[..., :DV], D ** -0.5, (slots >= 0).unsqueeze(1))
        lse[i] = l.transpose(0, 1)
    return out, lse


def _exact_sparse_prefill(st):
    s_q, h = st["case"]["s_q"], st["case"]["h_q"]
    out = torch.empty((s_q, h, DV), dtype=torch.float64, device=DEV)
    top = torch.empty((s_q, h), dtype=torch.float64, device=DEV)
    lse = torch.empty((s_q, h), dtype=torch.float64, device=DEV)
    kv = st["kv"].view(-1, D)
    for t0 in range(0, s_q, 128):
        t = slice(t0, min(t0 + 128, s_q))
        idx = st["indices"][t, 0].long()
        k = kv[idx.clamp(min=0)].double()
        out[t], l, m = _attend(st["q"][t].double(), k, k[..., :DV], D ** -0.5, (idx >= 0).unsqueeze(1))
        top[t], lse[t] = m / math.log(2), l / math.log(2)                          # base 2
    return out, top, lse


def _exact_mha(st):
    case = st["case"]
    q, k, v, d_out = st["q"].detach(), st["k"].detach(), st["v"].detach(), st.get("d_out")
    scale, group, lens = case["d_qk"] ** -0.5, case["h_q"] // case["h_k"], _lens(case)
    out = torch.empty((*q.shape[:2], 128), dtype=torch.float64, device=DEV)
    lse = torch.empty(q.shape[:2], dtype=torch.float64, device=DEV)
    dq, dk, dv = (torch.empty(x.shape, dtype=torch.float64, device=DEV) for x in (q, k, v))
    at = 0
    for n in lens:
        rows = slice(at, at + n)
        at += n
        visible = torch.ones((n, n), dtype=torch.bool, device=DEV).tril_() if case["causal"] else None
        for h in range(case["h_q"]):
            qh, kh, vh = q[rows, h].double(), k[rows, h // group].double(), v[rows, h // group].double()
            out[rows, h], lse[rows, h], _ = _attend(qh, kh, vh, scale, visible)
            if d_out is None:
                continue
            s = (qh @ kh.T).mul_(scale)
            if visible is not None:
                s.masked_fill_(~visible, -math.inf)
            p = s.sub_(lse[rows, h].unsqueeze(1)).exp_()
            g = d_out[rows, h].double()
            dv[rows, h] = p.T @ g
            ds = (g @ vh.T).sub_((g * out[rows, h]).sum(1, keepdim=True)).mul_(p)
            dq[rows, h], dk[rows, h] = (ds @ kh) * scale, (ds.T @ qh) * scale
    return (out, lse) if d_out is None else (out, lse, dq, dk, dv)
