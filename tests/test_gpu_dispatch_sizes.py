"""Dispatch at the sizes where its kernels change: the last batch that counts its
own layout and the first that gets a layout kernel, edges of the layout kernel's
warps, blocks and cluster, the route beyond it, batches of several rows per
block and their remainders; odd top-k (index pairs cannot be loaded) and repeats."""
import pytest
import torch

from mooncake_b200 import ep
from mooncake_b200.mooncake_ep_buffer import Buffer
from oracle import ep_oracle as ora
from tests.ep_harness import FakeGroup, make_rank_inputs
from tests.test_gpu_parity import _check_dispatch, _run_case

pytestmark = pytest.mark.gpu

SIZES = [  # T, H, E, K, fp8
    (1, 128, 8, 1, True), (1, 8320, 8, 1, False), (17, 640, 8, 1, False), (1001, 8320, 16, 1, False), (2, 8192, 8, 2, False), (3, 8320, 4, 3, True), (296, 512, 16, 3, True), (297, 512, 16, 3, False),
    (297, 1024, 256, 8, True), (300, 7168, 64, 16, False), (511, 128, 32, 5, True), (513, 2048, 4096, 2, False),
    (1023, 640, 24, 6, True), (1500, 8320, 8, 2, False), (2049, 384, 128, 8, True), (4096, 128, 4096, 4, False),
    (2341, 7168, 8, 8, False), (592, 4096, 16, 3, True), (593, 4096, 16, 3, False), (4096, 1024, 8, 2, True), (4097, 640, 8, 2, False), (8192, 128, 8, 1, True),
    (8192, 128, 256, 8, True), (8193, 128, 256, 8, True), (9001, 256, 16, 1, False),
    (400, 12416, 8, 8, False), (4800, 4096, 8, 8, False),
    (512, 4096, 8, 8, False), (513, 4096, 8, 8, True), (853, 8192, 4, 1, False), (854, 8192, 4, 1, False),  # marks for L2
    (1706, 4096, 8, 8, False), (1707, 4096, 8, 8, False),
    (199, 4096, 16, 8, True), (200, 4096, 16, 8, False), (292, 2816, 16, 8, True), (185, 4096, 16, 9, False),  # a group's counting
    (1036, 3584, 8, 2, False), (1037, 3584, 8, 2, False), (1481, 2688, 8, 8, False), (445, 4224, 8, 4, False),  # the two reduce kernels of a group
]


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("T,H,E,K,fp8", SIZES)
def test_dispatch_and_combine(T, H, E, K, fp8, staged):
    M = (T + 3) // 4 * 4
    x, idx, w = make_rank_inputs(11, 0, T, H, E, K, "zipf1.2" if T % 2 else "uniform", n_mask=T // 7)
    if K > 1:
        idx[::5, K - 1] = idx[::5, 0]  # an expert twice in one token's list
    if T > 4:
        idx[T // 2] = -1
    if staged and Buffer.get_ep_buffer_size_hint(M, H, 1, E) > 40e9:
        pytest.skip("needs more symmetric memory than a test should hold")
    buf = Buffer(FakeGroup(0, 1), Buffer.get_ep_buffer_size_hint(M, H, 1, E) if staged else 0)
    buf.runtime.set_option("force_staged", int(staged))
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    want = ora.dispatch([x], [idx], M, E, fp8)
    dx, di, dw = x.cuda(), idx.cuda(), w.cuda()
    for _ in range(2):  # both halves of the scratch
        recv, cnt, handle, _, _ = buf.dispatch(dx, di, active, M, E, 2_000_000, use_fp8=fp8)
        torch.cuda.synchronize()
        got = [dict(recv_x=recv[0] if fp8 else recv, scales=recv[1] if fp8 else None, recv_count=cnt, handle=handle)]
        if E * M * H <= 1 << 28:
            _check_dispatch(dict(R=1, E=E, M=M, fp8=fp8), got, want, None)
        else:
            assert torch.equal(cnt.cpu(), want[0]["recv_count"])
        if E * M * H <= 1 << 28:
            # combine, bit for bit: weights in listing order, every row from its own place
            y = torch.randn((E, M, H), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda",
                            dtype=torch.bfloat16)
            out, _, _ = buf.combine(y, di, dw, active, 2_000_000, handle)
            ref = ora.combine([y.cpu()], [idx], [w],
                              [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)[0]
            assert torch.equal(out.cpu().view(torch.int16), ref.view(torch.int16))
        if fp8:
            continue
        # the rows went where combine looks for them: x times the sum of the listed weights
        out, _, _ = buf.combine(recv, di, dw, active, 2_000_000, handle)
        ref = dx.float() * (dw * (di >= 0)).sum(dim=1, keepdim=True)
        assert float((out.float() - ref).abs().max() / ref.abs().max()) < 1e-2
    assert buf.runtime.status() == 0


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("T,H,E,K", [  # edges of the layout's words, chunks and loads of counts, and where it ends
    (31, 128, 8, 3), (33, 640, 8, 3), (127, 3584, 8, 5), (128, 4096, 300, 2), (129, 8320, 24, 16), (149, 7168, 8, 8),
    (2047, 128, 8, 4), (2049, 384, 64, 3), (600, 128, 2600, 1), (16384, 128, 8, 3), (16385, 128, 8, 3),
    (150, 128, 4096, 2), (2200, 128, 900, 3), (4300, 128, 300, 2),
    (301, 2048, 8, 1), (150, 2688, 16, 1), (149, 8320, 8, 1),  # four tiles of a row per warp (FP8), whole and not
    (149, 2560, 8, 4), (33, 3584, 16, 2), (150, 4480, 8, 3)])  # two, odd numbers of them
def test_positions_from_the_layout_kernel(T, H, E, K, fp8):
    """Positions looked up in bits and counts (or read, beyond them), repeats and empty tokens among them."""
    M = (T + 3) // 4 * 4
    x, idx, w = make_rank_inputs(17, 0, T, H, E, K, "zipf1.2", n_mask=T // 7)
    if K > 1:
        idx[::5, K - 1] = idx[::5, 0]
    buf = Buffer(FakeGroup(0, 1), 0)
    buf.runtime.set_option("fuse_layout", 0)
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    recv, cnt, handle, _, _ = buf.dispatch(x.cuda(), idx.cuda(), active, M, E, 2_000_000, use_fp8=fp8)
    got = [dict(recv_x=recv[0] if fp8 else recv, scales=recv[1] if fp8 else None, recv_count=cnt, handle=handle)]
    torch.cuda.synchronize()
    _check_dispatch(dict(R=1, E=E, M=M, fp8=fp8), got, ora.dispatch([x], [idx], M, E, fp8), None)
    y = torch.randn((E, M, H), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").to(torch.bfloat16)
    out, _, _ = buf.combine(y, idx.cuda(), w.cuda(), active, 2_000_000, handle)
    ref = ora.combine([y.cpu()], [idx], [w], [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)
    assert torch.equal(out.cpu().view(torch.int16), ref[0].view(torch.int16))
    assert buf.runtime.status() == 0


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("T,H,E,K,counted", [
    # several tokens per block and more of their tiles than the block has warps, ragged last batches
    (1001, 4096, 16, 1, True), (1481, 1152, 8, 2, True), (592, 4224, 8, 3, True), (591, 4480, 16, 3, True),
    # either side of where the layout kernel begins: 12 MB to one and two, 17 MB and a token per SM to more
    (1535, 4096, 8, 1, True), (1536, 4096, 8, 1, False), (767, 4096, 8, 2, True), (768, 4096, 8, 2, False),
    (271, 4096, 8, 8, True), (272, 4096, 8, 8, False), (297, 1664, 16, 16, True), (592, 128, 16, 16, True),
    (593, 128, 16, 16, False), (148, 8320, 8, 8, True), (149, 8320, 8, 8, False),
    # a token per block: one warp's tokens and more, several rounds of them, more tiles than warps, its end
    (1, 4224, 24, 16, True), (32, 128, 8, 5, True), (33, 640, 4096, 1, True), (129, 2048, 8, 3, True), (444, 128, 9, 8, True),
    (444, 4096, 16, 1, True), (445, 640, 9, 4, True), (147, 8704, 16, 7, True), (295, 4224, 8, 2, True), (296, 4224, 8, 2, True)])
def test_batches_that_count_for_themselves(T, H, E, K, counted, fp8):
    """Positions counted in the send kernel of a single rank, repeats and empty tokens among them, up to
    the sizes that it is used for; which kernel ran is looked up, so that the sizes follow the rule."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are those of 148 SMs")
    M = (T + 3) // 4 * 4
    x, idx, w = make_rank_inputs(19, 0, T, H, E, K, "zipf1.2", n_mask=T // 7)
    if K > 1:
        idx[::5, K - 1] = idx[::5, 0]
    buf = Buffer(FakeGroup(0, 1), 0)
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    ep.set_kernel_timing(True)
    try:
        recv, cnt, handle, _, _ = buf.dispatch(x.cuda(), idx.cuda(), active, M, E, 2_000_000, use_fp8=fp8)
    finally:
        ep.set_kernel_timing(False)
    torch.cuda.synchronize()
    assert any("layout" in name for name in ep.drain_kernel_times()) == (not counted)
    got = [dict(recv_x=recv[0] if fp8 else recv, scales=recv[1] if fp8 else None, recv_count=cnt, handle=handle)]
    _check_dispatch(dict(R=1, E=E, M=M, fp8=fp8), got, ora.dispatch([x], [idx], M, E, fp8), None)
    y = torch.randn((E, M, H), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").to(torch.bfloat16)
    out, _, _ = buf.combine(y, idx.cuda(), w.cuda(), active, 2_000_000, handle)
    ref = ora.combine([y.cpu()], [idx], [w], [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)
    assert torch.equal(out.cpu().view(torch.int16), ref[0].view(torch.int16))
    assert buf.runtime.status() == 0


@pytest.mark.parametrize("mode", ["hook", "sync"])
@pytest.mark.parametrize("T,fp8", [((280, 320), True), ((320, 280, 257), False), ((296, 297), False)])
def test_ranks_on_either_side_of_the_counting_limit(T, fp8, mode):
    """In-process groups: one rank counts its layout in the send kernel, another has a layout kernel."""
    _run_case(dict(R=len(T), tokens=list(T), M=320, H=128, E=8 * len(T), K=16, fp8=fp8, seed=3), mode=mode)


@pytest.mark.parametrize("mode", ["hook", "sync"])
@pytest.mark.parametrize("T,H,fp8", [((150, 250), 4096, False), ((150, 250), 4096, True), ((1, 294, 186), 4096, False)])
def test_ranks_of_one_launch_differ_in_bytes(T, H, fp8, mode):
    """In-process groups: ranks of up to two tokens per SM share a launch, however many bytes each of them sends."""
    _run_case(dict(R=len(T), tokens=list(T), M=296, H=H, E=8 * len(T), K=8, fp8=fp8, seed=5), mode=mode)


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("T", [0, 1, 40, 296])
def test_a_layout_kernel_for_small_batches(T, staged):
    """Option "fuse_layout" 0: the layout comes from a kernel of its own, with the same results."""
    H, E, K, M = 640, 16, 3, 300
    x, idx, w = make_rank_inputs(13, 0, T, H, E, K, n_mask=T // 7)
    buf = Buffer(FakeGroup(0, 1), Buffer.get_ep_buffer_size_hint(M, H, 1, E) if staged else 0)
    buf.runtime.set_option("force_staged", int(staged))
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    want = ora.dispatch([x], [idx], M, E, True)
    for fuse in (1, 0):
        buf.runtime.set_option("fuse_layout", fuse)
        ep.set_kernel_timing(True)
        try:
            recv, cnt, handle, _, _ = buf.dispatch(x.cuda(), idx.cuda(), active, M, E, 2_000_000)
        finally:
            ep.set_kernel_timing(False)
        torch.cuda.synchronize()
        assert any("layout" in name for name in ep.drain_kernel_times()) == (not fuse and T > 0)
        _check_dispatch(dict(R=1, E=E, M=M, fp8=True),
                        [dict(recv_x=recv[0], scales=recv[1], recv_count=cnt, handle=handle)], want, None)
        y = torch.randn((E, M, H), device="cuda").to(torch.bfloat16)
        out, _, _ = buf.combine(y, idx.cuda(), w.cuda(), active, 2_000_000, handle)
        ref = ora.combine([y.cpu()], [idx], [w], [dict(src_info=handle[0].cpu(), layout_range=handle[1].cpu())], M, E)
        assert torch.equal(out.cpu().view(torch.int16), ref[0].view(torch.int16))
    assert buf.runtime.status() == 0


@pytest.mark.parametrize("T,H", [(320, 4096), (1024, 7168)])  # the two reduce kernels of a group
def test_a_result_is_the_callers_until_its_hook_runs(T, H):
    """Work between combine and its hook may still read the result's memory, also work that lets the next kernel
    start early (a dispatch of these rows); without a hook the phases of a call overlap."""
    E = K = 8
    x, idx, w = (t.cuda() for t in make_rank_inputs(23, 0, T, H, E, K))
    buf = Buffer(FakeGroup(0, 1), Buffer.get_ep_buffer_size_hint(T, H, 1, E))
    buf.runtime.set_option("force_staged", 1)
    other = Buffer(FakeGroup(0, 1), 0)
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    recv, _, handle, _, _ = buf.dispatch(x, idx, active, T, E, 2_000_000, use_fp8=False)
    want, _, _ = buf.combine(recv, idx, w, active, 2_000_000, handle)
    for _ in range(4):
        recv, _, handle, _, hook = buf.dispatch(x, idx, active, T, E, 2_000_000, use_fp8=False, return_recv_hook=True)
        hook()
        out = torch.full((T, H), 7.0, dtype=torch.bfloat16, device="cuda")
        _, _, hook = buf.combine(recv, idx, w, active, 2_000_000, handle, return_recv_hook=True, out=out)
        between, count, _, _, _ = other.dispatch(out, idx, active, T, E, 2_000_000, use_fp8=False)
        hook()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        assert all(bool((between[e, :n] == 7).all()) for e, n in enumerate(count.tolist()))
    assert buf.runtime.status() == 0


@pytest.mark.parametrize("T", [2, 150])
def test_rows_of_more_blocks_than_are_resident(T):
    """Rows so long that one alone is shared by more combine blocks than the device holds at a time."""
    H, E, K = 128 * 18952, 2, 2
    x = torch.randn((T, H), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").to(torch.bfloat16)
    idx = torch.tensor([[0, 1]] * T, device="cuda")
    w = torch.full((T, K), 0.5, device="cuda")
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    buf = Buffer(FakeGroup(0, 1), 0)
    recv, _, handle, _, _ = buf.dispatch(x, idx, active, T, E, 2_000_000, use_fp8=False)
    out, _, _ = buf.combine(recv, idx, w, active, 2_000_000, handle)
    assert torch.equal(recv[0], x) and torch.equal(recv[1], x) and torch.equal(out, x)


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("T,M", [(5, 1 << 29), (700, 1 << 29), (700, (1 << 31) // 8)])
def test_tensors_of_2_to_the_31_rows(T, M, fp8):
    """Rows whose number has more than 31 bits. No device holds such tensors whole: every token names the
    last expert, whose part alone is there, and the bases that are passed lie that far ahead of it."""
    H, E, K = 128, 8, 2
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda").to(torch.bfloat16)
    idx = torch.tensor([[-1, E - 1], [E - 1, E - 1], [-1, -1], [E - 1, E]], device="cuda").repeat(T, 1)[:T].contiguous()
    sent = (idx == E - 1).any(dim=1).nonzero().flatten()
    n, width = len(sent), H if fp8 else 2 * H
    rows = torch.zeros((T, width), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((T,), dtype=torch.float32, device="cuda")  # (a scale per row: H is 128)
    src = torch.full((T,), -1, dtype=torch.int32, device="cuda")
    count, layout = (torch.full((E,), -1, dtype=d, device="cuda") for d in (torch.int32, torch.int64))
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    ahead, stream = (E - 1) * M, torch.cuda.current_stream().cuda_stream
    buf = ep.Buffer(0, 1, 0)
    for fuse in (1, 0):
        buf.set_option("fuse_layout", fuse)
        buf.dispatch(x.data_ptr(), idx.data_ptr(), active.data_ptr(), T, H, K, M, E, 2_000_000, fp8,
                     rows.data_ptr() - ahead * width, scales.data_ptr() - ahead * 4 if fp8 else 0, count.data_ptr(),
                     src.data_ptr() - ahead * 4, layout.data_ptr(), False, False, stream)
        torch.cuda.synchronize()
        assert count.tolist() == [0] * (E - 1) + [n] and layout.tolist() == count.tolist()
        assert torch.equal(src[:n].long(), sent) and bool((src[n:] == -1).all())
        want = ora.dispatch([x.cpu()], [idx.cpu()], (T + 3) // 4 * 4, E, fp8)[0]
        assert torch.equal(rows[:n].cpu(), want["recv_x"][E - 1, :n].contiguous().view(torch.uint8))
        if fp8:
            assert torch.equal(scales[:n].cpu(), want["scales"][E - 1, :n].flatten())
    y = torch.randn((T, H), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.rand((T, K), generator=g, device="cuda")
    out = torch.full((T, H), 7.0, dtype=torch.bfloat16, device="cuda")
    buf.combine(y.data_ptr() - ahead * 2 * H, idx.data_ptr(), w.data_ptr(), src.data_ptr() - ahead * 4, layout.data_ptr(),
                active.data_ptr(), E, T, H, K, M, E, 2_000_000, False, out.data_ptr(), False, False, stream)
    torch.cuda.synchronize()
    acc = torch.zeros((T, H), device="cuda", dtype=torch.float64)
    for k in range(K):
        at = (idx[sent, k] == E - 1).double() * w[sent, k].double()
        acc[sent] += at.unsqueeze(1) * y[:n].double()
    # (an fp32 sum of two products and one rounding to bf16: half a step, and both sums' errors)
    assert bool(((out.double() - acc).abs() <= acc.abs() * 2 ** -8 + 1e-6).all())
    assert buf.status() == 0
