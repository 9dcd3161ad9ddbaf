"""The native part of the Python binding: what it does not take itself (masks of
another length, wrong types and shapes) still ends in the wrapper's own checks."""
import pytest
import torch

from mooncake_b200 import Buffer
from oracle import ep_oracle as ora
from tests.ep_harness import FakeGroup, make_rank_inputs

pytestmark = pytest.mark.gpu

T, H, E, K, M = 12, 256, 8, 2, 16


def _layer(buf, dev, active, fp8=False, **kw):
    x, idx, w = dev
    recv, cnt, handle, _, _ = buf.dispatch(x, idx, active, M, E, 200_000, use_fp8=fp8)
    y = torch.nan_to_num((recv[0] if fp8 else recv).float()).to(torch.bfloat16)
    out, _, _ = buf.combine(y, idx, w, active, 200_000, handle, **kw)
    return y, cnt, handle, out


@pytest.mark.parametrize("mask", ["ones", "none", "other_length"])
def test_masks_and_caller_owned_output(mask):
    ins = make_rank_inputs(5, 0, T, H, E, K, n_mask=2)
    dev = [t.cuda() for t in ins]
    active = {"ones": torch.ones(1, dtype=torch.int32, device="cuda"), "none": None,
              "other_length": torch.zeros(3, dtype=torch.int32, device="cuda")}[mask]
    buf = Buffer(FakeGroup(0, 1), 0)
    buf._warned_active_ranks = True
    mine = torch.empty((T, H), dtype=torch.bfloat16, device="cuda")
    y, cnt, handle, out = _layer(buf, dev, active, out=mine)
    assert out is mine and handle[2:] == (M, H, E)
    want = ora.dispatch([ins[0]], [ins[1]], M, E, False)[0]
    assert torch.equal(cnt.cpu(), want["recv_count"])
    ref = ora.combine([y.cpu()], [ins[1]], [ins[2]],
                      [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)[0]
    assert torch.equal(out.cpu().view(torch.int16), ref.view(torch.int16))


def test_wrong_arguments_raise_assertion_errors():
    dev = [t.cuda() for t in make_rank_inputs(5, 0, T, H, E, K)]
    x, idx, w = dev
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    buf = Buffer(FakeGroup(0, 1), 0)
    for bad in ((x.float(), idx, active, M), (x.t().contiguous().t(), idx, active, M), (x, idx.int(), active, M),
                (x, idx[:4], active, M), (x, idx, active, T - 1), (x, idx, active.long(), M)):
        with pytest.raises(AssertionError):
            buf.dispatch(*bad, E, 200_000, use_fp8=False)
    with pytest.raises(AssertionError):
        buf.dispatch(x, idx, active, 15, E, 200_000)  # FP8: the rows of an expert come in fours
    with pytest.raises(RuntimeError, match="E > 0"):
        buf.dispatch(x, idx, active, M, 0, 200_000)
    with pytest.raises(RuntimeError, match="async_finish"):
        buf.dispatch(x, idx, active, M, E, 200_000, async_finish=True, return_recv_hook=True)
    y, _, handle, _ = _layer(buf, dev, active)
    for bad in ((y[:4], idx, w), (y, idx, w.half()), (y, idx[:3], w), (y.float(), idx, w)):
        with pytest.raises(AssertionError):
            buf.combine(*bad, active, 200_000, handle)
    with pytest.raises(AssertionError):
        buf.combine(y, idx, w, active, 200_000, handle, out=torch.empty((T, H), device="cuda"))
    with pytest.raises(TypeError, match="unexpected"):
        buf.runtime.dispatch(*([0] * 17), wrong=1)
    assert buf.runtime.status() == 0


def test_tensors_in_pinned_host_memory():
    """Everything but the rows of dispatch may lie in host memory that the device can reach."""
    from mooncake_b200 import ElasticBuffer
    ins = make_rank_inputs(6, 0, T, H, E, K, n_mask=2)
    x, (idx, w) = ins[0].cuda(), [t.pin_memory() for t in ins[1:]]
    active = torch.ones(1, dtype=torch.int32).pin_memory()
    mine = torch.empty((T, H), dtype=torch.bfloat16).pin_memory()
    buf = Buffer(FakeGroup(0, 1), 0)
    recv, cnt, handle, _, _ = buf.dispatch(x, idx, active, M, E, 200_000, use_fp8=False)
    y = torch.nan_to_num(recv.float()).to(torch.bfloat16)
    want = ora.dispatch([ins[0]], [ins[1]], M, E, False)[0]
    assert torch.equal(cnt.cpu(), want["recv_count"])
    ref = ora.combine([y.cpu()], [ins[1]], [ins[2]],
                      [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)[0]
    held = tuple(t.cpu().pin_memory() for t in handle[:2]) + handle[2:]
    for rows, h, out in ((y, handle, None), (y.cpu().pin_memory(), held, mine)):
        got, _, _ = buf.combine(rows, idx, w, active, 200_000, h, out=out)
        torch.cuda.synchronize()
        assert torch.equal(got.cpu().view(torch.int16), ref.view(torch.int16))
    for bad in ((x, ins[1], active), (ins[0], idx, active), (x, idx, torch.ones(1, dtype=torch.int32))):
        with pytest.raises(AssertionError):  # memory that the device cannot reach
            buf.dispatch(*bad, M, E, 200_000, use_fp8=False)
    ebuf = ElasticBuffer(FakeGroup(0, 1), num_max_tokens_per_rank=M, hidden=H, num_topk=K)
    erecv, _, ew, eh, _ = ebuf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, num_max_tokens_per_rank=M)
    there = (ins[1] >= 0).any(dim=1)
    assert torch.equal(erecv.cpu(), ins[0][there]) and torch.equal(ew.cpu(), ins[2][there])
    out, _, _ = ebuf.combine(erecv, eh)
    assert torch.equal(out.cpu(), ins[0] * there.unsqueeze(1))


def test_what_is_not_a_number_or_a_flag_is_refused():
    x, idx, w = [t.cuda() for t in make_rank_inputs(5, 0, T, H, E, K)]
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    buf = Buffer(FakeGroup(0, 1), 0)
    for bad in (dict(timeout_us=None), dict(num_max_dispatch_tokens_per_rank=None), dict(num_experts=None),
                dict(async_finish=None)):
        kw = dict(dict(num_max_dispatch_tokens_per_rank=M, num_experts=E, timeout_us=200_000, async_finish=False), **bad)
        with pytest.raises(TypeError):
            buf.dispatch(x, idx, active, use_fp8=False, **kw)
    for at in (3, 8, 9, 15, 17):
        args = [0] * 18
        args[at] = None
        with pytest.raises(TypeError):
            buf.runtime.dispatch(*args)
        with pytest.raises(TypeError):
            buf.runtime.combine(*(args if at in (8, 15, 17) else [0] * 13 + [None] + [0] * 4))
    recv, _, handle, _, hook = buf.dispatch(x, idx, active, M, E, 200_000, use_fp8=False, return_recv_hook=True)
    for bad in ((1,), dict(again=True)):
        with pytest.raises(TypeError):
            hook(*bad) if isinstance(bad, tuple) else hook(**bad)
    hook()
    _, event, _ = buf.combine(recv, idx, w, active, 200_000, handle, async_finish=True)
    event.event.current_stream_wait(stream_ptr=torch.cuda.current_stream().cuda_stream)
    with pytest.raises(TypeError):
        event.event.current_stream_wait()
    torch.cuda.synchronize()


def test_outputs_are_filled_where_torch_is_asked_to():
    """Under deterministic algorithms torch.empty fills its tensors; so do the calls' outputs."""
    from mooncake_b200 import ElasticBuffer
    x, idx, w = [t.cuda() for t in make_rank_inputs(5, 0, T, H, E, K)]
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    buf = Buffer(FakeGroup(0, 1), 0)
    ebuf = ElasticBuffer(FakeGroup(0, 1), num_max_tokens_per_rank=M, hidden=H, num_topk=K)
    zeros = [torch.zeros(1 << 20, device="cuda") for _ in range(8)]
    del zeros  # (blocks that the outputs may get: what is not written reads as zeros)
    torch.use_deterministic_algorithms(True)
    try:
        recv, cnt, handle, _, _ = buf.dispatch(x, idx, active, M, E, 200_000, use_fp8=False)
        erecv, eidx, ew, eh, _ = ebuf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E,
                                               num_max_tokens_per_rank=M, do_cpu_sync=False)
    finally:
        torch.use_deterministic_algorithms(False)
    n = cnt.tolist()
    assert all(bool(recv[e, n[e]:].isnan().all()) and bool((handle[0][e, n[e]:] == -1).all()) for e in range(E))
    assert torch.equal(erecv[:T], x) and bool(erecv[T:].isnan().all()) and bool(ew[T:].isnan().all())
