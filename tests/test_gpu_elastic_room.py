"""Expanded elastic calls whose aligned segments end beyond the rows that the expanded
tensors have room for (tokens of the group * top-k): the tensors stay inside their memory,
the rows beyond are dropped and reported."""
import pytest
import torch

from mooncake_b200 import ElasticBuffer
from oracle import elastic_oracle as eo
from tests.ep_harness import FakeGroup, make_rank_inputs

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
