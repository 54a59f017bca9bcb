"""Calls that the paths for ranks of one process have to refuse on the host, before anything is launched, and forms of a call that
they have to go on taking."""
import ctypes as C

import pytest

import cann_hccl_b200 as H
from cann_hccl_b200 import _lib as L

PER_RANK = ("rows", "pos", "dstRow", "expertOffsets", "recvRows", "overflow")


@pytest.fixture(scope="module")
def pair():
    c = H.Communicator.init_local(2, device=False)
    yield c
    c.destroy()


def moe_call(comm, missing=None, rank=1, entry="dispatch", instead=None):
    """A dispatch or combine of the host communicator's ranks, with one entry of one table null (or moved by `instead` bytes):
    result code.  Complete tables come as far as the check of the transport (the launches need a GPU)."""
    mem = C.create_string_buffer(64)
    at = (C.addressof(mem) + 31) // 32 * 32
    odd = None if instead is None else at + instead
    y = L.MoeLayer(tokens=4, capacityRows=8, topk=2, hidden=8, nExperts=4, scratch=at)
    call = {n: (C.c_void_p * 2)(at, at) for n in ("x", "idx", "gates", "out", "given")}
    for n in PER_RANK:
        for r in range(2):
            getattr(y, n)[r] = at
    if missing == "scratch":
        y.scratch = None
    elif missing in PER_RANK:
        getattr(y, missing)[rank] = odd
    elif missing:
        call[missing][rank] = odd
    if entry == "dispatch":
        return L.lib().HcclB200MoeDispatchLocal(comm.handle, C.byref(y), call["x"], call["idx"], None)
    rows = call["given"] if missing == "given" else None
    return L.lib().HcclB200MoeCombineLocal(comm.handle, C.byref(y), rows, call["idx"], call["gates"], call["out"], None)


def test_moe_tables_with_a_null_entry(pair):
    for entry, tables in (("dispatch", ("x", "idx")), ("combine", ("idx", "gates", "out", "given"))):
        assert moe_call(pair, entry=entry) == L.E_NOT_SUPPORT
        for name in PER_RANK + ("scratch",) + tables:
            for rank in range(2):
                assert moe_call(pair, name, rank, entry) == L.E_PTR, (entry, name, rank)


def test_moe_rows_off_their_boundaries(pair):
    """Rows move in 16-byte vectors, experts and gates in words: an address between is refused (32-byte vectors are a choice)."""
    for entry, rows, words in (("dispatch", ("rows", "x"), ("idx",)), ("combine", ("rows", "out"), ("idx", "gates")), ("combine", ("given", "out"), ())):
        for name in rows:
            for off, want in ((2, L.E_PARA), (8, L.E_PARA), (16, L.E_NOT_SUPPORT)):
                assert moe_call(pair, name, 1, entry, off) == want, (entry, name, off)
        for name in words:
            for off, want in ((2, L.E_PARA), (4, L.E_NOT_SUPPORT)):
                assert moe_call(pair, name, 0, entry, off) == want, (entry, name, off)


@pytest.mark.parametrize("nlocal,bad", [(1, None), (1, [None]), (2, [None, None])])
def test_moe_call_path_refuses_none(nlocal, bad):
    """The Python call path, for a lone rank (which passes its buffer without a list) and for several: no communicator is reached."""
    import numpy as np
    good = [np.zeros(8, np.float32) for _ in range(nlocal)]
    L.lib()
    with pytest.raises(TypeError):
        L.fast.moe_dispatch(0, nlocal, 0, bad, good, 0)
    with pytest.raises(TypeError):
        L.fast.moe_dispatch(0, nlocal, 0, good, bad, 0)
    for at in range(3):
        args = [good, good, good]
        args[at] = bad
        with pytest.raises(TypeError):
            L.fast.moe_combine(0, nlocal, 0, 0, *args, 0)
    assert L.fast.moe_combine(0, nlocal, 0, 0, good, good, good, 0) == L.E_PTR  # all buffers there: refused for the communicator


def test_tensor_parallel_layers_with_a_null_entry(pair):
    """Complete tables come as far as the check of the transport."""
    mem = C.create_string_buffer(64)
    at = C.addressof(mem)
    lib = L.lib()
    calls = {"gather": lambda t: lib.HcclB200AllGatherMatmul(pair.handle, *t, 256, 256, 64, None),
             "gather_act": lambda t: lib.HcclB200AllGatherMatmulAct(pair.handle, *t, 256, 256, 64, 1, None),
             "scatter": lambda t: lib.HcclB200MatmulReduceScatter(pair.handle, *t, 256, 256, 64, None)}
    for name, call in calls.items():
        assert call([(C.c_void_p * 2)(at, at) for _ in range(3)]) == L.E_NOT_SUPPORT
        for table in range(3):
            for rank in range(2):
                t = [(C.c_void_p * 2)(at, at) for _ in range(3)]
                t[table][rank] = None
                assert call(t) == L.E_PTR, (name, table, rank)


def test_combine_before_any_dispatch():
    pytest.importorskip("torch")
    from cann_hccl_b200.parallel import moe
    ex = object.__new__(moe.MoEExchange)
    ex._topk = None
    with pytest.raises(RuntimeError):
        ex.combine(None)


def test_closed_exchange():
    pytest.importorskip("torch")
    from cann_hccl_b200.parallel import moe

    class Memory:
        freed = []

        def mem_free(self, handle):
            self.freed.append(handle)

    ex = object.__new__(moe.MoEExchange)
    ex.comm, ex.h_recv, ex.h_out, ex._topk = Memory(), 1, 2, [object()]
    ex.recv = ex.expert_out = [object()]
    ex.close()
    assert ex.comm.freed == [1, 2]
    with pytest.raises(RuntimeError):
        ex.dispatch(None, None)
    with pytest.raises(RuntimeError):
        ex.combine(None)


@pytest.mark.parametrize("device", [False, pytest.param(True, marks=pytest.mark.gpu)])
def test_alltoallv_counts_are_compared_on_every_call(device):
    """More calls than ranks of other processes would compare: a sender's count above the receiver's would run over the
    receiver's next block."""
    import numpy as np
    if device:
        torch = pytest.importorskip("torch")
        if not torch.cuda.is_available():
            pytest.skip("no GPU")
    p, n = 3, 5
    c = H.Communicator.init_local(p, device=device, device_id=0) if device else H.Communicator.init_local(p, device=False)
    ins = [np.arange(p * n, dtype=np.float32) + 100 * r for r in range(p)]
    outs = [np.full(p * (n + 1), -1, np.float32) for _ in range(p)]
    if device:
        ins, outs = [torch.from_numpy(x).cuda() for x in ins], [torch.from_numpy(x).cuda() for x in outs]
    host = lambda x: x.cpu().numpy() if device else x
    sc = np.full((p, p), n, np.uint64)
    sd = np.tile(np.arange(p, dtype=np.uint64) * np.uint64(n), (p, 1))
    rd = np.tile(np.arange(p, dtype=np.uint64) * np.uint64(n + 1), (p, 1))
    for _ in range(20):
        c.all_to_all_v(ins, sc, sd, outs, np.ascontiguousarray(sc.T), rd)
    if device:
        assert c.sync() == 0
    before = [host(o).copy() for o in outs]
    assert all(b[q * (n + 1)] == 100 * q + r * n and b[q * (n + 1) + n] == -1 for r, b in enumerate(before) for q in range(p))
    for i, j, sent, expected in ((0, 2, n + 1, n), (2, 0, n, n + 1)):
        m, want = sc.copy(), sc.T.copy()
        m[i, j], want[j, i] = sent, expected
        with pytest.raises(H.HcclError) as e:
            c.all_to_all_v(ins, m, sd, outs, want, rd)
        assert e.value.code == L.E_PARA
    assert all(np.array_equal(b, host(o)) for b, o in zip(before, outs))
    assert c.destroy() == L.SUCCESS


def test_collectives_with_a_null_buffer(pair):
    """A rank without a buffer that the collective reads or writes is refused; one that the rank does not need may be missing."""
    import numpy as np
    n = 6
    x, big = [np.ones(n, np.float32) for _ in range(2)], [np.zeros(2 * n, np.float32) for _ in range(2)]
    need = {L.ALLREDUCE: (x, x), L.ALLGATHER: (x, big), L.REDUCE_SCATTER: (big, x), L.ALLTOALL: (x, big), L.BROADCAST: (x, x), L.REDUCE: (x, x),
            L.SCATTER: (big, x), L.GATHER: (x, big)}
    spare = {L.BROADCAST: {("send", 1), ("recv", 0)}, L.REDUCE: {("recv", 1)}, L.SCATTER: {("send", 1)}, L.GATHER: {("recv", 1)}}
    for coll, (send, recv) in need.items():
        for side in ("send", "recv"):
            for rank in range(2):
                if (side, rank) in spare.get(coll, ()):
                    continue
                s, r = list(send), [y.copy() for y in recv]
                (s if side == "send" else r)[rank] = None
                with pytest.raises(H.HcclError) as e:
                    pair.collective(coll, s, r, 3, L.FP32, root=0)
                assert e.value.code == L.E_PTR, (coll, side, rank)
    out = [np.zeros(n, np.float32), None]                       # only the root receives
    pair.reduce(x, out, 0)
    assert np.array_equal(out[0], 2 * x[0])
    zero, at = np.zeros(2, np.uint64), np.array([3, 5], np.uint64)
    pair.collective(L.ALLGATHER_V, [None, None], [None, None], 0, L.FP32, counts=zero, displs=at)
    pair.collective(L.REDUCE_SCATTER_V, [None, None], [None, None], 0, L.FP32, counts=zero, displs=at)
    c = np.array([[0, 2], [0, 0]], np.uint64)
    d = np.zeros((2, 2), np.uint64)
    got = [None, np.zeros(2, np.float32)]                       # rank 0 only sends, rank 1 only receives
    pair.all_to_all_v([x[0], None], c, d, got, np.ascontiguousarray(c.T), d)
    assert np.array_equal(got[1], x[0][:2])
    for send, recv in (([None, x[0]], got), ([x[0], None], [x[0], None])):
        with pytest.raises(H.HcclError) as e:
            pair.collective(L.ALLTOALLV, send, recv, 0, L.FP32, rows=(c, d, np.ascontiguousarray(c.T), d))
        assert e.value.code == L.E_PTR


def test_buffers_as_rows_of_one_array(pair):
    """One array with a row per rank is a list of buffers too; the number of rows has to be the number of ranks."""
    import numpy as np
    x, y = np.arange(10, dtype=np.float32).reshape(2, 5), np.zeros((2, 5), np.float32)
    pair.collective(L.ALLREDUCE, x, y, 5, L.FP32)
    assert np.array_equal(y, np.stack([x.sum(0)] * 2))
    torch = pytest.importorskip("torch")
    tx, ty = torch.arange(10.).reshape(2, 5), torch.zeros(2, 5)
    pair.collective(L.ALLREDUCE, tx, ty, 5, L.FP32)
    assert torch.equal(ty, tx.sum(0).repeat(2, 1))
    for call, count in (("all_reduce", 5), ("all_gather", 5), ("reduce_scatter", 4), ("all_to_all", 4)):  # a row's count, not the array's
        src = np.arange(16, dtype=np.float32).reshape(2, 8)[:, :count if call != "reduce_scatter" else 8].copy()
        dst = np.full((2, 16), -1, np.float32)[:, :{"all_reduce": 5, "all_gather": 10, "reduce_scatter": 4, "all_to_all": 4}[call]].copy()
        lists = [d.copy() for d in dst]
        getattr(pair, call)(src, dst)
        getattr(pair, call)(list(src), lists)
        assert np.array_equal(dst, np.stack(lists)) and (dst >= 0).all()
    for bad in (x[:1], [x[0]], (x[0], x[0], x[1])):
        with pytest.raises(AssertionError):
            pair.collective(L.ALLREDUCE, bad, y, 5, L.FP32)


def test_buffer_lists_that_are_not_what_they_say(pair):
    """A list that shrinks while its buffers are asked for their addresses, a sequence whose length is not its items."""
    import numpy as np
    x = np.zeros(4, np.float32)

    class Shrinks:
        def __init__(self, of):
            self.of = of

        def data_ptr(self):
            del self.of[1:]
            return x.ctypes.data

    class Short:
        def __len__(self):
            return 2

        def __iter__(self):
            return iter([x])

    shrinking = []
    shrinking += [Shrinks(shrinking), x]
    for bad in (shrinking, Short()):
        with pytest.raises(AssertionError):
            pair.collective(L.ALLREDUCE, bad, [x, x.copy()], 4, L.FP32)


def test_direct_kernels_by_name_need_one_gpu(pair):
    """The algorithm of ranks that share a process and a GPU, asked for by its number: not on CPU ranks."""
    import numpy as np
    assert L.ALGO_NAMES[L.ALGO_LOCAL] == "local" and L.lib().HcclB200AlgoName(L.ALGO_LOCAL) == b"local"
    x, y = [np.ones(4, np.float32) for _ in range(2)], [np.zeros(4, np.float32) for _ in range(2)]
    with pytest.raises(H.HcclError) as e:
        pair.all_reduce(x, y, algo=L.ALGO_LOCAL)
    assert e.value.code == L.E_NOT_SUPPORT
    pair.all_reduce(x, y)
    assert pair.trace()[-1]["algo"] != "local" and np.array_equal(y[0], x[0] * 2)
