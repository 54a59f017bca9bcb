"""MoE exchange of all ranks in one process: the launches that serve every rank at once, and the per-rank launches that
communicators over several processes take, against the plain PyTorch statement."""
import pytest

torch = pytest.importorskip("torch")
import cann_hccl_b200 as H  # noqa: E402
from cann_hccl_b200 import _lib as L  # noqa: E402
from cann_hccl_b200.parallel import moe  # noqa: E402

pytestmark = pytest.mark.gpu


# tokens x top-k around the chunk of 1024 pairs and beyond 32 chunks; top-k around the batch of eight rows; rows shorter than a
# CTA, and longer than its four vectors per thread.  One CTA, clusters of two to eight, and more pairs or counters than they take.  CTAs of the
# combine that take four and two tokens, the last one fewer
@pytest.mark.parametrize("p,T,hidden,E,k", [(1, 1, 8, 4, 1), (1, 127, 264, 16, 8), (2, 129, 256, 64, 8), (3, 257, 2048, 33, 9), (4, 100, 8456, 8, 2),
                                            (1, 4100, 64, 256, 8), (8, 40, 512, 128, 17), (2, 33, 9216, 8, 2), (1, 1025, 16, 256, 8), (2, 512, 16, 1500, 8),
                                            (4, 700, 32, 1024, 8), (8, 1024, 16, 32, 8), (1, 8300, 16, 64, 8), (3, 911, 2816, 48, 3), (8, 20, 16, 2048, 4), (1, 2371, 2816, 16, 2), (2, 593, 40, 16, 4)])
@pytest.mark.parametrize("per_rank", [False, True])
def test_exchange(p, T, hidden, E, k, per_rank):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    cfg = L.CommConfig.default()
    cfg.hcclBufferSize = 2
    c = H.Communicator.init_local(p, device=True, device_id=0, config=cfg)
    ex = moe.MoEExchange(c, T, hidden, E, k, capacity_factor=float(p))
    assert ex._layer is not None
    if per_rank:
        ex._layer = None
    g = torch.Generator(device="cuda").manual_seed(T)
    xs = [torch.randn(T, hidden, device="cuda", generator=g).to(torch.bfloat16) for _ in range(p)]
    idx, gates = map(list, zip(*[moe.route(T, E, k, 7, r) for r in range(p)]))
    idx[0][0, 0] = -1                                            # a slot without an expert is skipped
    launches = c.stats()["launches"]
    for _ in range(2):                                            # the second call finds the scratch as the first left it
        ex.dispatch(xs if p > 1 else xs[0], idx if p > 1 else idx[0])
        assert c.sync() == 0, c.describe_status()
        El = E // p
        for r in range(p):
            want = torch.stack([sum((idx[s] == r * El + e).sum() for s in range(p)) for e in range(El)])
            offs = ex.expert_offsets[r].long()
            assert torch.equal(offs[1:] - offs[:-1], want) and int(offs[0]) == 0
            assert int(ex.recv_rows[r]) == int(want.sum()) and int(ex.overflow[r]) == 0
            for s in range(p):                                    # every pair's row is where dst_row says, and rows are not shared
                mine = (idx[s] >= r * El) & (idx[s] < (r + 1) * El)
                rows = ex.dst_row[s].view(T, k)[mine].long()
                assert torch.equal(ex.recv[r][rows], xs[s].repeat_interleave(mine.sum(1), dim=0))
            taken = torch.cat([ex.dst_row[s].view(T, k)[(idx[s] >= r * El) & (idx[s] < (r + 1) * El)] for s in range(p)])
            assert taken.unique().numel() == taken.numel()
            ex.expert_out[r].copy_(-ex.recv[r])
        outs = ex.combine(gates if p > 1 else gates[0])
        same = ex.combine(gates if p > 1 else gates[0], source="recv")
        assert c.sync() == 0, c.describe_status()
        outs, same = (outs, same) if p > 1 else ([outs], [same])
        for r in range(p):
            want = xs[r].float() * (gates[r] * (idx[r] >= 0)).sum(1, keepdim=True)
            # k products summed in fp32 (batches of eight are rounded to bf16 in between on the per-rank path), one bf16 rounding
            tol = 2.0 ** -8 * (1 + (k - 1) // 8)
            assert bool(((same[r].float() - want).abs() <= tol * xs[r].float().abs() + 1e-6).all())
            assert torch.equal(outs[r], -same[r])
    # two dispatches of two launches and four combines of one; per rank: an all-gather (or its direct copy) and barriers each time
    assert c.stats()["launches"] == launches + 8 if not per_rank else c.stats()["launches"] > launches
    ex.close()
    c.destroy()


def test_rows_beyond_the_capacity_are_dropped():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = H.Communicator.init_root(1, H.Communicator.get_root_info(), 0, device=True)
    T, hidden, E, k = 256, 64, 8, 2
    ex = moe.MoEExchange(c, T, hidden, E, k, capacity_factor=0.5)
    guard = ex.expert_out[0].fill_(3)
    x = torch.randn(T, hidden, device="cuda").to(torch.bfloat16)
    idx, gates = moe.route(T, E, k, 7, 0)
    ex.dispatch(x, idx)
    out = ex.combine(gates, source="recv")
    assert c.sync() == 0
    assert int(ex.overflow[0]) == 1 and int(ex.recv_rows[0]) == T * k
    kept = (ex.dst_row[0].view(T, k) < ex.cap).float()
    want = x.float() * (gates * kept).sum(1, keepdim=True)
    assert bool(((out.float() - want).abs() <= 2.0 ** -8 * x.float().abs() + 1e-6).all())
    assert bool((guard == 3).all())
    ex.close()
    c.destroy()


@pytest.mark.parametrize("p,T,hidden,E,k", [(1, 128, 2048, 64, 8), (4, 128, 7168, 256, 8), (1, 8300, 64, 64, 8), (2, 4200, 512, 16, 8)])
def test_inputs_rewritten_in_place(p, T, hidden, E, k):
    """Activations and experts get new values at the same addresses, by kernels on the same stream right before every dispatch:
    the rows that arrive are the new ones (numbered by one cluster, and through global memory).  No host wait in between."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    cfg = L.CommConfig.default()
    cfg.hcclBufferSize = 2
    c = H.Communicator.init_local(p, device=True, device_id=0, config=cfg)
    ex = moe.MoEExchange(c, T, hidden, E, k, capacity_factor=float(p))
    xs = [torch.zeros(T, hidden, device="cuda", dtype=torch.bfloat16) for _ in range(p)]
    idx = [torch.zeros(T, k, device="cuda", dtype=torch.int32) for _ in range(p)]
    kinds = [[(torch.randn(T, hidden, device="cuda").to(torch.bfloat16), moe.route(T, E, k, 11 + v, r)[0]) for r in range(p)] for v in range(3)]
    good = torch.zeros(24, device="cuda", dtype=torch.bool)
    El = E // p
    torch.cuda.synchronize()
    for it in range(good.numel()):
        for r, (x, i) in enumerate(kinds[it % 3]):
            torch.add(x, 0, out=xs[r])
            idx[r].copy_(i)
        ex.dispatch(xs if p > 1 else xs[0], idx if p > 1 else idx[0])
        same = []
        for r, (x, i) in enumerate(kinds[it % 3]):
            rows = ex.dst_row[r].view(T, k).long()
            got = torch.stack(ex.recv)[(i // El).long(), rows]
            same.append((got == x[:, None, :]).all())
        good[it] = torch.stack(same).all()
    assert c.sync() == 0, c.describe_status()
    assert bool(good.all()), good.nonzero().flatten().tolist()
    ex.close()
    c.destroy()


def test_first_dispatch_on_another_stream():
    """The exchange is made while its stream is busy and used on another one at once: the numbering of more pairs than one cluster
    takes needs the scratch zero from the start."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    T, hidden, E, k = 8300, 64, 64, 8
    c = H.Communicator.init_root(1, H.Communicator.get_root_info(), 0, device=True)
    x = torch.randn(T, hidden, device="cuda").to(torch.bfloat16)
    idx, gates = moe.route(T, E, k, 5, 0)
    side = torch.cuda.Stream()
    words = L.lib().HcclB200MoeScratchBytes(1, T, k, E) // 4
    torch.full((words,), 7, device="cuda", dtype=torch.int32)  # what the allocator hands out next is not zero by chance
    torch.cuda.synchronize()
    torch.cuda._sleep(50_000_000)
    ex = moe.MoEExchange(c, T, hidden, E, k)
    with torch.cuda.stream(side):
        ex.dispatch(x, idx)
        out = ex.combine(gates, source="recv")
    side.synchronize()
    assert int(ex.recv_rows[0]) == T * k and torch.equal(ex.recv[0][ex.dst_row[0].view(T, k).long()], x[:, None].expand(T, k, hidden))
    assert bool(((out.float() - x.float()).abs() <= 2.0 ** -8 * x.float().abs() + 1e-6).all())
    ex.close()
    c.destroy()
