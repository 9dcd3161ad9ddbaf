"""The work a user of this package has it do on one GPU, as cases that can be timed.

Four ways into the package:

  buffer   `Buffer.dispatch` / `Buffer.combine` (mooncake_b200/mooncake_ep_buffer.py): what an MoE layer
           calls; the package allocates the packed tensors of every call.
  native   `ep.Buffer.dispatch` / `.combine` (mooncake_b200/ep.py) with device pointers: what a wrapper of
           its own calls (Mooncake's own Python wrapper does), on output tensors that the caller keeps.
  group    `Buffer` on the path that a rank of a multi-GPU group takes: receive rows in symmetric memory,
           counts, answers and payload words exchanged (option "force_staged"; the one rank talks to itself).
  elastic  `ElasticBuffer.dispatch` / `.combine`: flat receive rows, cached handles, expanded layout.

One pass is one layer's exchange: dispatch, then combine. Between them stand the experts, which are not the
package's work: with bf16 payloads the received rows themselves go back (identity experts), with FP8 payloads
the experts' outputs are tensors made in advance. Sizes are those of bench.py's workloads and of the tests,
and ragged ones around them. Everything that a call defines is returned. Rows of the packed tensors that no
token was sent to are undefined, so where the package allocates those tensors (`buffer`, `group`) the
received rows come back through combine; where the caller does (`native`), they come back whole.
"""
import math

import numpy as np
import torch

from mooncake_b200 import Buffer, ElasticBuffer, ep

TIMEOUT_US = 2_000_000


class _OneRank:
    """A process group of one rank, as far as the package looks at it."""

    def rank(self):
        return 0

    def size(self):
        return 1


def _layer(name, api, T, M, H, E, K, fp8, routing, masked=0.0, mode="plain"):
    return dict(name=name, api=api, tokens=T, max_tokens=M, hidden=H, experts=E, topk=K, fp8=fp8,
                routing=routing, masked=masked, mode=mode)


def _elastic(name, T, H, E, K, routing, training, expand, cpu_sync, masked=0.0):
    return dict(name=name, api="elastic", tokens=T, max_tokens=T, hidden=H, experts=E, topk=K, fp8=False,
                routing=routing, masked=masked, mode="plain", training=training, expand=expand,
                cpu_sync=cpu_sync)


def listed():
    return [
        # a single sequence being decoded: one token, DeepSeek-V3-shaped layer, FP8 (the package's default)
        _layer("decode_1_token", "buffer", 1, 128, 7168, 256, 8, True, "uniform"),
        # bench.py's default: a decode batch of 128 tokens of the same layer
        _layer("decode_128_fp8", "buffer", 128, 128, 7168, 256, 8, True, "uniform"),
        # Qwen3-shaped decode under skewed routing, driven by a wrapper that keeps its own output tensors
        _layer("decode_256_zipf_fp8", "native", 256, 256, 4096, 128, 8, True, "zipf"),
        # a small model in bf16 (bench.py's c1)
        _layer("small_model_bf16", "buffer", 128, 128, 2048, 16, 4, False, "softmax"),
        # Mixtral-shaped batch of a ragged size with padding tokens (-1), overlapped through async_finish
        _layer("mixtral_1000_async", "buffer", 1000, 1024, 4096, 8, 2, False, "uniform", 0.05, "async"),
        # prefill of 4096 tokens in bf16 (bench.py's c3), the bandwidth-bound end
        _layer("prefill_4096_bf16", "buffer", 4096, 4096, 7168, 256, 8, False, "uniform"),
        # Qwen3-shaped prefill chunk of an odd size in FP8, skewed routing, caller-owned tensors
        _layer("prefill_2001_zipf_fp8", "native", 2001, 2048, 4096, 128, 8, True, "zipf"),
        # one rank's decode call on the multi-GPU path
        _layer("group_decode_128_fp8", "group", 128, 128, 7168, 256, 8, True, "uniform"),
        # a prefill chunk on the multi-GPU path with send and receive phases apart (two micro-batches overlap)
        _layer("group_1024_hook", "group", 1024, 1024, 4096, 128, 8, False, "uniform", 0.0, "hook"),
        # elastic-style inference call: no CPU sync, decode batch
        _elastic("elastic_decode_128", 128, 7168, 256, 8, "uniform", False, False, False),
        # a training step of one layer: dispatch and combine forward, then backward, where the gradient of
        # combine is a dispatch with the cached handle and the gradient of dispatch is a combine
        _elastic("elastic_training_4096", 4096, 7168, 256, 8, "softmax", True, False, True),
        # the expanded (expert-major) layout that a grouped GEMM reads, with padding tokens
        _elastic("elastic_expand_1024", 1024, 4096, 128, 8, "uniform", False, True, True, 0.05),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["bytes"] for c in listed())
    while True:
        api = rng.choice(["buffer", "buffer", "native", "group", "elastic"])
        T = _between(rng, 1, 4096)
        H = 128 * _between(rng, 4, 56)
        E = rng.choice([8, 16, 32, 64, 96, 128, 160, 256])
        K = rng.choice([k for k in (1, 2, 4, 6, 8) if k <= E])
        routing = rng.choice(["uniform", "softmax", "zipf"])
        masked = rng.choice([0.0, 0.0, 0.05])
        if api == "elastic":
            training, expand = rng.random() < 0.4, rng.random() < 0.3
            cpu_sync = expand or rng.random() < 0.6
            # (rows that are received by no one stay undefined where the host does not learn how many there are)
            known = cpu_sync and not training
            c = _elastic("", T, H, E, K, routing, training, expand, cpu_sync, masked if known else 0.0)
        else:
            M = T if T % 4 == 0 and rng.random() < 0.5 else 128 * -(-T // 128)
            c = _layer("", api, T, M, H, E, K, rng.random() < 0.5, routing, masked,
                       rng.choice(["plain", "plain", "async", "hook"]))
        del c["name"]
        # a packed tensor and the symmetric buffer have room for every token at every expert
        packed = E * c["max_tokens"] * H
        room = {"buffer": 4e9, "native": 1.2e9, "group": 8e8, "elastic": math.inf}[api]
        if packed <= room and work(c)["bytes"] <= most:
            return c


def _padded(case):
    """Tokens that only fill the batch up: no expert in their lists."""
    return int(case["tokens"] * case["masked"])


def _routing(case, g):
    T, E, K = case["tokens"], case["experts"], case["topk"]
    scores = torch.randn((T, E), generator=g, device="cuda")
    if case["routing"] == "softmax":
        scores = torch.softmax(scores, dim=-1)
    elif case["routing"] == "zipf":  # Zipf(1.2) over the experts, without replacement (Gumbel top-k)
        logp = -1.2 * torch.log(torch.arange(1, E + 1, dtype=torch.float32, device="cuda"))
        u = torch.rand((T, E), generator=g, device="cuda").clamp(min=1e-20)
        scores = logp - torch.log(-torch.log(u))
    weights, idx = torch.topk(scores, K, dim=-1)
    if case["masked"]:
        idx[torch.randperm(T, generator=g, device="cuda")[:_padded(case)]] = -1
    if case["routing"] == "softmax":
        weights = weights / weights.sum(dim=-1, keepdim=True)
    else:
        weights = torch.softmax(torch.rand((T, K), generator=g, device="cuda"), dim=-1)
    return idx.to(torch.int64).contiguous(), weights.float().contiguous()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, M, H, E, K = (case[k] for k in ("tokens", "max_tokens", "hidden", "experts", "topk"))
    s = dict(case)
    s["x"] = torch.randn((T, H), generator=g, device="cuda", dtype=torch.bfloat16)
    s["idx"], s["weights"] = _routing(case, g)
    s["active"] = torch.ones(1, dtype=torch.int32, device="cuda")
    if case["api"] == "elastic":
        s["buf"] = ElasticBuffer(_OneRank(), num_max_tokens_per_rank=M, hidden=H, num_topk=K)
        s["grad"] = torch.randn((T, H), generator=g, device="cuda", dtype=torch.bfloat16)
        for _ in range(2):  # a program's buffer has been warmed up: the scratch of both calls in flight is there
            _run_elastic(s)
            torch.cuda.synchronize()
        return s
    if case["fp8"] or case["api"] == "native":  # the experts' outputs
        s["y"] = torch.empty((E, M, H), dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    if case["api"] != "native":
        group = case["api"] == "group"
        s["buf"] = Buffer(_OneRank(), Buffer.get_ep_buffer_size_hint(M, H, 1, E) if group else 0)
        if group:
            s["buf"].runtime.set_option("force_staged", 1)
        return s
    s["buf"] = ep.Buffer(0, 1, 0)
    zeros = lambda shape, dtype: torch.zeros(shape, dtype=dtype, device="cuda")  # noqa: E731
    s["recv_x"] = zeros((E, M, H), torch.uint8 if case["fp8"] else torch.bfloat16)
    s["scales"] = zeros((E, H // 128, M), torch.float32) if case["fp8"] else None
    s["count"], s["src_info"] = zeros((E,), torch.int32), zeros((E, M), torch.int32)
    s["layout"], s["combined"] = zeros((E, 1), torch.int64), zeros((T, H), torch.bfloat16)
    return s


def _finish(mode, event, hook):
    if mode == "async":
        event.current_stream_wait()
    elif mode == "hook":
        hook()


def _run_buffer(s):
    buf, mode = s["buf"], s["mode"]
    how = dict(async_finish=mode == "async", return_recv_hook=mode == "hook")
    recv, count, handle, event, hook = buf.dispatch(
        s["x"], s["idx"], s["active"], s["max_tokens"], s["experts"], TIMEOUT_US, use_fp8=s["fp8"], **how)
    _finish(mode, event, hook)
    combined, event, hook = buf.combine(s["y"] if s["fp8"] else recv, s["idx"], s["weights"], s["active"],
                                        TIMEOUT_US, handle, **how)
    _finish(mode, event, hook)
    return combined, count, handle[1]


def _run_native(s):
    buf, mode = s["buf"], s["mode"]
    is_async, is_hook = mode == "async", mode == "hook"
    stream = torch.cuda.current_stream().cuda_stream
    T, M, H, E, K = s["tokens"], s["max_tokens"], s["hidden"], s["experts"], s["topk"]
    idx, active = s["idx"].data_ptr(), s["active"].data_ptr()
    src_info, layout = s["src_info"].data_ptr(), s["layout"].data_ptr()
    event, hook = buf.dispatch(s["x"].data_ptr(), idx, active, T, H, K, M, E, TIMEOUT_US, s["fp8"],
                               s["recv_x"].data_ptr(), s["scales"].data_ptr() if s["fp8"] else 0,
                               s["count"].data_ptr(), src_info, layout, is_async, is_hook, stream)
    if is_async:
        event.current_stream_wait(stream)
    elif is_hook:
        hook()
    event, hook = buf.combine(s["y"].data_ptr(), idx, s["weights"].data_ptr(), src_info, layout, active, E, T,
                              H, K, M, E, TIMEOUT_US, False, s["combined"].data_ptr(), is_async, is_hook, stream)
    if is_async:
        event.current_stream_wait(stream)
    elif is_hook:
        hook()
    return s["recv_x"], s["scales"], s["count"], s["src_info"], s["layout"], s["combined"]


def _run_elastic(s):
    buf = s["buf"]
    recv_x, recv_idx, recv_weights, handle, _ = buf.dispatch(
        s["x"], topk_idx=s["idx"], topk_weights=s["weights"], num_experts=s["experts"],
        num_max_tokens_per_rank=s["max_tokens"], do_expand=s["expand"], do_cpu_sync=s["cpu_sync"])
    out, _, _ = buf.combine(recv_x, handle)
    metadata = handle.recv_src_metadata if s["expand"] else handle.recv_src_metadata[:, :2]
    got = [recv_x, recv_idx, recv_weights, metadata, handle.psum_num_recv_tokens_per_scaleup_rank,
           handle.psum_num_recv_tokens_per_expert, handle.dst_buffer_slot_idx, out]
    if s["cpu_sync"]:  # the host's copy of the counts, as a launcher of grouped GEMMs wants it
        got.append(np.array(handle.num_recv_tokens_per_expert_list, dtype=np.int32))
    if s["training"]:
        recv_grad, _, _, again, _ = buf.dispatch(s["grad"], handle=handle)
        grad_x, _, _ = buf.combine(recv_grad, again)
        got += [recv_grad, grad_x]
    return got


def run(state):
    return {"buffer": _run_buffer, "group": _run_buffer, "native": _run_native,
            "elastic": _run_elastic}[state["api"]](state)


def work(case):
    """Inputs read once, outputs written once; combine's weighted sums."""
    T, H, E, K = (case[k] for k in ("tokens", "hidden", "experts", "topk"))
    n = T - _padded(case)
    sent = n * K  # (token, expert) selections
    if case["api"] == "elastic":
        rows = sent if case["expand"] else n  # a token travels once
        forward = (2 * H * T + 12 * T * K + 2 * H * rows + 12 * n * K + 8 * n + 12 * T * K  # dispatch
                   + 2 * H * rows + 2 * H * T)  # combine
        backward = 2 * (2 * H * T + 2 * H * rows) if case["training"] else 0
        passes = 2 if case["training"] else 1
        return {"bytes": forward + backward, "flops": 1.0 * passes * H * rows}
    payload = H + 4 * (H // 128) if case["fp8"] else 2 * H
    dispatch = 2 * H * T + 8 * T * K + sent * (payload + 4) + 12 * E
    combine = 2 * H * sent + 12 * T * K + 2 * H * T
    return {"bytes": dispatch + combine, "flops": 2.0 * sent * H}


def tolerance(case):
    """Whole numbers, FP8 bytes and bf16 rows that are only moved are the same in any implementation. Combine
    sums in fp32 and rounds to bf16 once: another order of the sum may move a value by one bf16 step."""
    return {"rel": 4e-3, "max": 0.02}
