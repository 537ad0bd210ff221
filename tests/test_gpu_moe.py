"""MoE dispatch (all-to-all + permute) and combine (all-to-all + weighted sum) kernels,
run as an emulated world on one GPU and checked against a PyTorch fp32 reference."""
import pytest
import torch

from flagcx_b200 import capi
from flagcx_b200.parallel.moe import MoeDispatcher, route

pytestmark = pytest.mark.gpu


def _sorted_rows(rows: torch.Tensor) -> torch.Tensor:
    """Rows in lexicographic order of their exact bit patterns, so that two tensors hold the
    same multiset of rows exactly when the results are equal element for element."""
    bits = rows.contiguous().view(torch.int16).to(torch.int64).cpu()
    order = list(range(bits.shape[0]))
    order.sort(key=lambda i: bits[i].tolist())
    return bits[order]


# dedup: a token crosses NVLink once per destination rank (1) or once per expert (0);
# reduce: the expert rank adds up a token's weighted outputs (1) or the owner pulls every row (0)
@pytest.mark.parametrize("dedup,reduce", [(1, 1), (1, 0), (0, 1), (0, 0)])
@pytest.mark.parametrize("n,T,H,E,K", [(2, 33, 128, 8, 2), (4, 64, 256, 16, 4), (8, 96, 512, 64, 8), (2, 70, 128, 4, 4),
                                       (4, 24, 2688, 32, 8)])  # 336 vectors: 2 turns of a copy, 6 of a combine, the last in part
def test_dispatch_groups_rows_by_expert_and_combine_weights_them(n, T, H, E, K, dedup, reduce, monkeypatch):
    monkeypatch.setenv("FLAGCX_MOE_DEDUP", str(dedup))
    monkeypatch.setenv("FLAGCX_MOE_COMBINE_REDUCE", str(reduce))
    comms = capi.Comm.emu_world(n, 0)
    try:
        epr = E // n
        cap = T * K * n  # worst case: everything lands on one rank
        moes = [MoeDispatcher(comms[r], T, H, K, E, cap) for r in range(n)]
        g = torch.Generator().manual_seed(0)
        xs = [torch.randn(T, H, generator=g).to(torch.bfloat16).cuda() for _ in range(n)]
        routed = [route(torch.randn(T, E, generator=g).cuda(), K) for _ in range(n)]
        for r in range(n):
            moes[r].dispatch(xs[r], routed[r][0])
        torch.cuda.synchronize()
        for c in comms:
            assert c.async_error() == 0, c.last_error()
        # rows of local expert le on rank d: tokens of rank 0 first, then rank 1, ...
        for d in range(n):
            offs = moes[d].expert_offsets.cpu().tolist()
            for le in range(epr):
                e = d * epr + le
                want_rows = []
                for s in range(n):
                    sel = (routed[s][0] == e).any(dim=1).cpu()
                    rows = xs[s].cpu()[sel]
                    got = moes[d].recv_rows[offs[le] + len(want_rows): offs[le] + len(want_rows) + rows.shape[0]].cpu()
                    # order inside one (source, expert) group is arbitrary: compare whole rows as
                    # multisets (rows sorted lexicographically, then element for element)
                    assert torch.equal(_sorted_rows(got), _sorted_rows(rows)), (d, e, s)
                    want_rows.extend([None] * rows.shape[0])
                assert offs[le + 1] - offs[le] == len(want_rows)
            # the "expert": scale every row of expert e by (e + 1)
            for le in range(epr):
                e = d * epr + le
                moes[d].expert_out[offs[le]:offs[le + 1]] = (moes[d].recv_rows[offs[le]:offs[le + 1]].float() * (e + 1)).to(torch.bfloat16)
        outs = [torch.empty(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(n)]
        for r in range(n):
            moes[r].combine(routed[r][1], outs[r])
        torch.cuda.synchronize()
        for c in comms:
            assert c.async_error() == 0, c.last_error()
        for r in range(n):
            idx, w = routed[r]
            scale = (w * (idx.float() + 1)).sum(1, keepdim=True)  # sum_k w_k (e_k + 1)
            ref = xs[r].float() * scale
            err = ((outs[r].float() - ref).abs() / ref.abs().clamp(min=1.0)).max().item()
            assert err < 0.03, (r, err)
        for m in moes:
            m.close()
    finally:
        capi.Comm.emu_world_destroy(comms)


def test_capacity_overflow_is_reported_not_written():
    n, T, H, E, K = 2, 32, 64, 4, 2
    comms = capi.Comm.emu_world(n, 0)
    try:
        moes = [MoeDispatcher(comms[r], T, H, K, E, 8) for r in range(n)]  # far too small
        xs = [torch.randn(T, H).to(torch.bfloat16).cuda() for _ in range(n)]
        idx = torch.zeros(T, K, dtype=torch.int32, device="cuda")
        idx[:, 1] = 1  # everything to rank 0
        for r in range(n):
            moes[r].dispatch(xs[r], idx)
        torch.cuda.synchronize()
        assert comms[0].async_error() == capi.flagcxInvalidArgument
    finally:
        capi.Comm.emu_world_destroy(comms)


# more tokens than a CTA's table holds (256), more groups than it looks at in one turn, rows that
# end inside a piece (257 vectors: pieces of 160 and 97) and inside a round of the combine
@pytest.mark.parametrize("T,H,ctas", [(1, 8, 3), (256, 64, 1), (257, 64, 1), (600, 264, 2), (31, 2056, 1)])
@pytest.mark.parametrize("reduce", [1, 0])
def test_few_ctas_and_ragged_rows(T, H, ctas, reduce, monkeypatch):
    monkeypatch.setenv("FLAGCX_MOE_CTAS", str(ctas))
    monkeypatch.setenv("FLAGCX_MOE_COMBINE_REDUCE", str(reduce))
    n, E, K = 2, 8, 5
    comms = capi.Comm.emu_world(n, 0)
    try:
        moes = [MoeDispatcher(comms[r], T, H, K, E, T * K * n) for r in range(n)]
        g = torch.Generator().manual_seed(T)
        for t in (T, max(1, T // 3), T):  # a second batch of another size, and a third
            xs = [torch.randn(t, H, generator=g).to(torch.bfloat16).cuda() for _ in range(n)]
            routed = [route(torch.randn(t, E, generator=g).cuda(), K) for _ in range(n)]
            for r in range(n):
                moes[r].dispatch(xs[r], routed[r][0])
            for m in moes:
                offs = m.expert_offsets.cpu().tolist()
                for le in range(E // n):
                    scale = moes.index(m) * (E // n) + le + 1
                    m.expert_out[offs[le]:offs[le + 1]] = (m.recv_rows[offs[le]:offs[le + 1]].float() * scale).to(torch.bfloat16)
            outs = [torch.full((t, H), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(n)]
            for r in range(n):
                moes[r].combine(routed[r][1], outs[r])
            torch.cuda.synchronize()
            assert all(c.async_error() == 0 for c in comms)
            for r in range(n):
                idx, w = routed[r]
                ref = xs[r].float() * (w * (idx.float() + 1)).sum(1, keepdim=True)
                # all summands have one sign, so the three roundings to 8 significant bits (the expert's,
                # the pre-reduced row's, the result's) change the result by 2^-8 of its value each
                assert ((outs[r].float() - ref).abs() <= 3.02 * 2.0 ** -8 * ref.abs() + 1e-6).all()
        for m in moes:
            m.close()
    finally:
        capi.Comm.emu_world_destroy(comms)


# Four ranks of which two post: nothing is launched before the others have.  Both orders, in a new
# world and in one whose last operation was of the second kind.
@pytest.mark.parametrize("used", [False, True])
@pytest.mark.parametrize("first", ["dispatch", "all_reduce"])
def test_ranks_that_post_different_operations_are_refused(first, used):
    n, T, H, E, K = 4, 8, 64, 8, 2
    comms = capi.Comm.emu_world(n, 0)
    try:
        moes = [MoeDispatcher(comms[r], T, H, K, E, T * K * n) for r in range(n)]
        g = torch.Generator().manual_seed(1)
        xs = [torch.randn(T, H, generator=g).to(torch.bfloat16).cuda() for _ in range(n)]
        routed = [route(torch.randn(T, E, generator=g).cuda(), K) for _ in range(n)]
        outs = [torch.empty_like(x) for x in xs]
        post = {"dispatch": lambda r: moes[r].dispatch(xs[r], routed[r][0]),
                "all_reduce": lambda r: comms[r].all_reduce(xs[r], outs[r], T * H, capi.BFLOAT16)}
        second = "all_reduce" if first == "dispatch" else "dispatch"
        if used:
            for r in range(n):
                post[second](r)
        post[first](0)
        with pytest.raises(RuntimeError):
            post[second](1)
        for r in range(1, n):  # the others still complete what rank 0 has posted
            post[first](r)
        torch.cuda.synchronize()
        assert all(c.async_error() == 0 for c in comms)
        if first == "all_reduce":
            ref = sum(x.double() for x in xs)
            assert float((outs[2].double() - ref).abs().max()) < 0.05
        else:  # every row that was dispatched has arrived
            assert sum(int(m.expert_offsets[-1]) for m in moes) == n * T * K
        for m in moes:
            m.close()
    finally:
        capi.Comm.emu_world_destroy(comms)


# A lone rank has no barriers that would keep its layers apart: two of them on two streams, each with
# its own tokens and weights, over and over.
def test_two_layers_of_one_rank_at_the_same_time(monkeypatch):
    monkeypatch.setenv("FLAGCX_MOE_COMBINE_REDUCE", "0")
    comm = capi.Comm.init_rank(1, capi.get_unique_id(), 0)
    try:
        T, H, E, K = 700, 2048, 16, 4
        streams = [torch.cuda.Stream() for _ in range(2)]
        g = torch.Generator().manual_seed(5)
        layers = []
        for _ in streams:
            m = MoeDispatcher(comm, T, H, K, E, T * K)
            x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
            idx, w = route(torch.randn(T, E, generator=g).cuda(), K)
            layers.append((m, x, idx, w, torch.empty(20, T, H, dtype=torch.bfloat16, device="cuda")))
        for (m, x, idx, w, outs), s in zip(layers, streams):
            m.dispatch(x, idx)
            m.expert_out.copy_(m.recv_rows)
        torch.cuda.synchronize()
        for i in range(20):
            for (m, x, idx, w, outs), s in zip(layers, streams):
                m.combine(w, outs[i], stream=s)
        torch.cuda.synchronize()
        assert comm.async_error() == 0, comm.last_error()
        for m, x, idx, w, outs in layers:
            ref = x.float() * w.sum(1, keepdim=True)
            # fp32 sums of K products, rounded to bf16 once
            assert bool(((outs.float() - ref).abs() <= ref.abs() * 2 ** -8 + x.float().abs() * K * 2 ** -23).all())
            assert bool((outs == outs[0]).all())
            m.close()
    finally:
        comm.destroy()
