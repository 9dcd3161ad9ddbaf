"""Expanded elastic calls whose aligned segments end beyond the rows that the expanded
tensors have room for (tokens of the group * top-k): the tensors stay inside their memory,
the rows beyond are dropped and reported."""
import pytest
import torch

from mooncake_b200 import ElasticBuffer
from oracle import elastic_oracle as eo
from tests.ep_harness import FakeGroup, make_rank_inputs
from tests.test_gpu_elastic import _combine, _dispatch, _group

pytestmark = pytest.mark.gpu

SIZES = [  # T, H, E, K, alignment: counted in the copy kernel (two tokens per SM and less), behind a layout kernel
    (64, 256, 64, 8, 128), (16, 128, 256, 4, 128), (296, 640, 16, 3, 128), (1, 128, 8, 2, 64),
    (297, 256, 128, 8, 128), (700, 1152, 24, 2, 256), (2049, 128, 64, 1, 512),
]


def _inside_its_memory(t):
    if t.numel() == 0:
        return True
    last = t.storage_offset() + sum((n - 1) * s for n, s in zip(t.shape, t.stride()))
    return (last + 1) * t.element_size() <= t.untyped_storage().nbytes()


def _inputs(T, H, E, K):
    x, idx, w = make_rank_inputs(83, 0, T, H, E, K, "uniform", n_mask=T // 9)
    if T > 2:
        idx[T // 2] = -1
    return x, idx, w


@pytest.mark.parametrize("T,H,E,K,alignment", SIZES)
def test_dispatch_stays_inside_its_tensors(T, H, E, K, alignment):
    x, idx, w = _inputs(T, H, E, K)
    want = eo.elastic_dispatch([x], [idx], [w], E, T, alignment, True)[0]
    n, room = want["n"], T * K
    psum = want["psum_expert"].tolist()
    assert psum[E - 1] > room  # (else this tests nothing)
    buf = ElasticBuffer(FakeGroup(0, 1), num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    for sync in (True, False):
        recv, ridx, rw, h, _ = buf.dispatch(x.cuda(), topk_idx=idx.cuda(), topk_weights=w.cuda(), num_experts=E,
                                            num_max_tokens_per_rank=T, expert_alignment=alignment, do_expand=True,
                                            do_cpu_sync=sync)
        # before anything of them is touched
        assert all(_inside_its_memory(t) for t in (recv, ridx, rw, h.recv_src_metadata))
        assert recv.shape == (room, H) and rw.shape == (room,)
        torch.cuda.synchronize()
        assert h.psum_num_recv_tokens_per_expert.tolist() == psum
        if sync:
            assert h.num_recv_tokens_per_expert_list == [int(((idx == e).any(dim=1)).sum()) for e in range(E)]
        used = want["used"][:room]
        assert torch.equal(recv.cpu()[used].view(torch.int16), want["recv_x"][:room][used].view(torch.int16))
        assert torch.equal(rw.cpu()[used], want["recv_topk_weights"][:room][used])
        md = want["recv_src_metadata"].clone()
        md[:, 2:][md[:, 2:] >= room] = -1
        assert torch.equal(h.recv_src_metadata[:n].cpu(), md)
        assert buf.runtime.status() == 1  # rows out of range, nothing else


@pytest.mark.parametrize("T,H,E,K,alignment", SIZES)
def test_combine_adds_the_rows_that_there_was_room_for(T, H, E, K, alignment):
    x, idx, w = _inputs(T, H, E, K)
    want = eo.elastic_dispatch([x], [idx], [w], E, T, alignment, True)[0]
    room = T * K
    buf = ElasticBuffer(FakeGroup(0, 1), num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    for sync in (True, False):
        recv, _, _, h, _ = buf.dispatch(x.cuda(), topk_idx=idx.cuda(), num_experts=E, num_max_tokens_per_rank=T,
                                        expert_alignment=alignment, do_expand=True, do_cpu_sync=sync)
        y = torch.randn((room, H), generator=torch.Generator().manual_seed(T)).to(torch.bfloat16)
        for rows in (room, room // 2):  # a tensor with fewer rows is not read beyond them either
            out, _, _ = buf.combine(y[:rows].cuda(), h)
            ref = torch.zeros((T, H), dtype=torch.bfloat16)
            for (_, t), md in zip(want["rows"], want["recv_src_metadata"][:, 2:].tolist()):
                there = [y[v] for v in md if 0 <= v < rows]
                if there:
                    ref[t] = eo.bf16_sum(there)
            assert torch.equal(out.cpu().view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("Ts,M,H,E,K,alignment,staged", [
    ([33, 20], 40, 256, 32, 4, 128, True), ([64, 0], 64, 128, 8, 2, 256, True), ([9, 9], 9, 640, 4, 1, 64, True),
    ([40], 40, 256, 64, 8, 128, True), ([16385], 16385, 128, 4, 1, 8192, False)])
def test_general_path(Ts, M, H, E, K, alignment, staged):
    """Groups, and the batches that a single rank's own kernels do not take."""
    R, room = len(Ts), len(Ts) * M * K
    ins = [make_rank_inputs(89, r, Ts[r], H, E, K, "uniform", n_mask=3) for r in range(R)]
    xs, idxs, ws = [i[0] for i in ins], [i[1] for i in ins], [i[2] for i in ins]
    want = eo.elastic_dispatch(xs, idxs, ws, E, M, alignment, True)
    assert any(o["n_expanded"] > room for o in want)
    bufs = _group(R, M, H, K, staged)
    keep = []
    outs = _dispatch(bufs, xs, idxs, ws, E, M, alignment, True, keep)
    g = torch.Generator().manual_seed(M)
    ys = [torch.randn((room, H), generator=g).to(torch.bfloat16) for _ in range(R)]
    back = [{} for _ in range(R)]  # what a rank sends back for (source, token)
    for r, (d, o) in enumerate(zip(outs, want)):
        used = o["used"][:room]
        assert d["psum_expert"].tolist() == o["psum_expert"].tolist()
        assert torch.equal(d["recv_x"].cpu()[:used.shape[0]][used].view(torch.int16),
                           o["recv_x"][:room][used].view(torch.int16))
        assert torch.equal(d["recv_w"].cpu()[:used.shape[0]][used], o["recv_topk_weights"][:room][used])
        md = o["recv_src_metadata"].clone()
        md[:, 2:][md[:, 2:] >= room] = -1
        assert torch.equal(d["md"][:o["n"]].cpu(), md)
        assert bufs[r].runtime.status() == int(bool((o["recv_src_metadata"][:, 2:] >= room).any()))
        for key, rows in zip(o["rows"], md[:, 2:].tolist()):
            there = [ys[r][v] for v in rows if v >= 0]
            back[r][key] = eo.bf16_sum(there) if there else torch.zeros(H, dtype=torch.bfloat16)
    got = _combine(bufs, [y.cuda() for y in ys], outs, E, M, True)
    for s in range(R):
        for t in range(Ts[s]):
            lanes = eo.rank_lanes(idxs[s][t], E // R, E)
            order = [d for d, _ in sorted(lanes.items(), key=lambda kv: kv[1])]
            ref = eo.bf16_sum([back[d][(s, t)] for d in order]) if order else torch.zeros(H, dtype=torch.bfloat16)
            if t % max(1, Ts[s] // 200) == 0 or not order:
                assert torch.equal(got[s][t].cpu().view(torch.int16), ref.view(torch.int16)), (s, t)
