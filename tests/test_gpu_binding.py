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
