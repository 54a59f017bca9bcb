"""Direct collectives of communicators that hold every rank in this process on one GPU (algorithm left to the selector),
against a plain PyTorch reference: sizes around vectors and tiles, every alignment, in-place forms."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
import numpy as np  # noqa: E402
import cann_hccl_b200 as H  # noqa: E402
from cann_hccl_b200 import _lib as L  # noqa: E402

pytestmark = pytest.mark.gpu

# below a vector, around one vector, around a few tiles of 128 threads, many tiles (which hold as much as fills a thread's loads in
# the reductions; the copies' largest tile is test_large_copies)
SIZES = (1, 3, 17, 4095, 4097, 1_300_001)


@pytest.fixture(scope="module")
def comms():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    cache = {}

    def get(p):
        if p not in cache:
            cfg = L.CommConfig.default()
            cfg.hcclBufferSize = 2
            cache[p] = H.Communicator.init_local(p, device=True, device_id=0, config=cfg)
        return cache[p]

    yield get
    for c in cache.values():
        assert c.destroy() == L.SUCCESS


def rnd(p, n, dtype, seed, shift=lambda r: 0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for r in range(p):
        x = torch.rand(n + 16, device="cuda", generator=g) * 2 - 1
        x = x.to(dtype) if dtype.is_floating_point else (x * 4).to(dtype)
        out.append(x[shift(r):shift(r) + n])
    return out


def reduced(ins, op):
    acc = ins[0].double() if ins[0].dtype.is_floating_point else ins[0].clone()
    for x in ins[1:]:
        y = x.to(acc.dtype)
        acc = {L.SUM: acc + y, L.PROD: acc * y, L.MAX: torch.maximum(acc, y), L.MIN: torch.minimum(acc, y)}[op]
    return acc


def check(got, want, dtype, p):
    if not dtype.is_floating_point:
        assert torch.equal(got, want)
        return
    # p - 1 roundings of the accumulator (unit roundoff of fp32 / fp64), one of the result, values below p in magnitude
    eps = {torch.float64: 2.0 ** -52, torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert float((got.double() - want).abs().max()) <= p * p * eps


def done(c, algo="local"):
    assert c.sync() == 0, c.describe_status()
    assert c.trace()[-1]["algo"] == algo, c.trace()[-1]


@pytest.mark.parametrize("p", [2, 3, 4, 8, 11])
@pytest.mark.parametrize("dtype,op", [(torch.float32, L.SUM), (torch.bfloat16, L.SUM), (torch.float16, L.MAX), (torch.int8, L.MIN),
                                      (torch.int64, L.PROD), (torch.float64, L.SUM)])
def test_reductions(comms, p, dtype, op):
    c = comms(p)
    for n in SIZES:
        ins = rnd(p, n, dtype, n)
        outs = [torch.full_like(x, 9) for x in ins]
        c.all_reduce(ins, outs, op=op)
        done(c)
        want = reduced(ins, op)
        for o in outs:
            check(o, want, dtype, p)
        outs = [torch.full_like(x, 9) for x in ins]
        c.reduce(ins, outs, p - 1, op=op)
        done(c)
        check(outs[p - 1], want, dtype, p)
        assert all(bool((o == 9).all()) for o in outs[:-1])     # only the root's buffer is written
        m = max(1, n // p)
        ins = rnd(p, m * p, dtype, n + 1)                        # odd blocks start anywhere inside a vector
        outs = [torch.full((m,), 9, device="cuda", dtype=dtype) for _ in range(p)]
        c.reduce_scatter(ins, outs, op=op)
        done(c)
        want = reduced(ins, op)
        for r, o in enumerate(outs):
            check(o, want[r * m:(r + 1) * m], dtype, p)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.uint8])
@pytest.mark.parametrize("shift_in,shift_out", [(1, 0), (0, 1), (3, 3), (5, 2), (-1, 0), (0, -1)])
def test_alignments(comms, dtype, shift_in, shift_out):
    """Every rank's buffers at the same offset from a 16-byte boundary, or (negative) at a different one on each rank."""
    p, n = 4, 100_003
    c = comms(p)
    at = lambda s: (lambda r: s if s >= 0 else r * 3 % 7)
    ins = rnd(p, n, dtype, 5, at(shift_in))
    base = [torch.full((n + 32,), 9, device="cuda", dtype=dtype) for _ in range(p)]
    outs = [b[8 + at(shift_out)(r):8 + at(shift_out)(r) + n] for r, b in enumerate(base)]
    c.all_reduce(ins, outs, op=L.MAX)
    done(c)
    for o in outs:
        assert torch.equal(o.float(), reduced(ins, L.MAX).float())
    for r, b in enumerate(base):                                 # nothing around the output was touched
        lo = 8 + at(shift_out)(r)
        assert bool((b[:lo] == 9).all()) and bool((b[lo + n:] == 9).all())
    gbase = [torch.full((n * p + 32,), 9, device="cuda", dtype=dtype) for _ in range(p)]
    gout = [b[8 + at(shift_out)(r):8 + at(shift_out)(r) + n * p] for r, b in enumerate(gbase)]
    c.all_gather(ins, gout)
    done(c)
    for r, (o, b) in enumerate(zip(gout, gbase)):
        assert torch.equal(o, torch.cat(ins))
        lo = 8 + at(shift_out)(r)
        assert bool((b[:lo] == 9).all()) and bool((b[lo + n * p:] == 9).all())


@pytest.mark.parametrize("p", [2, 5])
def test_in_place(comms, p):
    c = comms(p)
    n = 70_001
    ins = rnd(p, n, torch.float32, 1)
    want = reduced(ins, L.SUM)
    c.all_reduce(ins, ins)
    done(c)
    for x in ins:
        check(x, want, torch.float32, p)
    ins = rnd(p, n * p, torch.float32, 2)
    want = reduced(ins, L.SUM)
    c.reduce_scatter(ins, [x[r * n:(r + 1) * n] for r, x in enumerate(ins)])
    done(c)
    for r, x in enumerate(ins):
        check(x[r * n:(r + 1) * n], want[r * n:(r + 1) * n], torch.float32, p)
    full = rnd(p, n * p, torch.float32, 3)
    blocks = [x[r * n:(r + 1) * n].clone() for r, x in enumerate(full)]
    c.all_gather([x[r * n:(r + 1) * n] for r, x in enumerate(full)], full)
    done(c)
    for x in full:
        assert torch.equal(x, torch.cat(blocks))


@pytest.mark.parametrize("p", [2, 4, 9])
def test_copies(comms, p):
    c = comms(p)
    for n in SIZES:
        n = min(n, 100_003)
        bufs = rnd(p, n, torch.float32, n)
        want = bufs[p - 1].clone()
        c.broadcast(bufs, p - 1)
        done(c)
        assert all(torch.equal(b, want) for b in bufs)
        big, small = rnd(p, n * p, torch.bfloat16, n), [torch.zeros(n, device="cuda", dtype=torch.bfloat16) for _ in range(p)]
        c.scatter(big, small, 1)
        done(c)
        assert torch.equal(torch.cat(small), big[1])
        back = [torch.zeros_like(x) for x in big]
        c.gather(small, back, 0)
        done(c)
        assert torch.equal(back[0], big[1])
        out = [torch.zeros_like(x) for x in big]
        c.all_to_all(big, out)
        done(c)
        for r in range(p):
            assert torch.equal(out[r], torch.cat([big[q][r * n:(r + 1) * n] for q in range(p)]))


def test_variable_counts(comms):
    p = 4
    c = comms(p)
    counts, displs = np.array([5, 0, 4101, 33], np.uint64), np.array([0, 8, 16, 4200], np.uint64)
    total = 4300
    ins = [rnd(1, max(1, int(counts[r])), torch.float32, r)[0] for r in range(p)]
    outs = [torch.full((total,), 9.0, device="cuda") for _ in range(p)]
    c.all_gather_v(ins, outs, counts, displs)
    done(c)
    want = torch.full((total,), 9.0, device="cuda")
    for r in range(p):
        want[int(displs[r]):int(displs[r] + counts[r])] = ins[r][:int(counts[r])]
    assert all(torch.equal(o, want) for o in outs)
    rin = rnd(p, total, torch.float32, 9)
    rout = [torch.full((5000,), 9.0, device="cuda") for _ in range(p)]
    c.reduce_scatter_v(rin, rout, counts, displs)
    done(c)
    ref = reduced(rin, L.SUM)
    for r in range(p):
        k = int(counts[r])
        if k:
            check(rout[r][:k], ref[int(displs[r]):int(displs[r]) + k], torch.float32, p)
        assert bool((rout[r][k:] == 9).all())
    c.barrier()
    assert c.sync() == 0


class At:
    """A buffer by its address: what a C caller passes."""

    def __init__(self, t, off):
        self.t, self.off = t, off

    def data_ptr(self):
        return self.t.data_ptr() + self.off


@pytest.mark.parametrize("dtype,code", [(torch.float32, L.FP32), (torch.bfloat16, L.BFP16), (torch.float64, L.FP64)])
@pytest.mark.parametrize("off_in,off_out", [((1, 1, 1), (0, 0, 0)), ((0, 0, 0), (1, 1, 1)), ((3, 1, 0), (0, 0, 0)), ((1, 2, 3), (5, 5, 5)), ((0, 1, 0), (1, 0, 3))])
def test_reductions_of_buffers_inside_an_element(comms, dtype, code, off_in, off_out):
    """Addresses that are no multiples of the element's size, on all ranks or on some: byte copies made them a matter of speed
    on the kernels that stage."""
    p = 3
    c = comms(p)
    es = torch.empty(0, dtype=dtype).element_size()
    for n in (1, 37, 40_003):
        ins = rnd(p, n * p, dtype, n)
        mem = [torch.zeros(n * p * es + 64, device="cuda", dtype=torch.uint8) for _ in range(p)]
        out = [torch.full((n * p * es + 64,), 9, device="cuda", dtype=torch.uint8) for _ in range(p)]
        for m, x, o in zip(mem, ins, off_in):
            m[16 + o:16 + o + n * p * es] = x.view(torch.uint8)
        send, recv = [At(m, 16 + o) for m, o in zip(mem, off_in)], [At(m, 16 + o) for m, o in zip(out, off_out)]
        for coll, count, mine in ((L.ALLREDUCE, n * p, lambda r: slice(0, n * p)), (L.REDUCE_SCATTER, n, lambda r: slice(r * n, (r + 1) * n))):
            for m in out:
                m.fill_(9)
            c.collective(coll, send, recv, count, code, op=L.MAX)
            done(c)
            want = reduced(ins, L.MAX)
            for r, (m, o) in enumerate(zip(out, off_out)):
                assert torch.equal(m[16 + o:16 + o + count * es].clone().view(dtype).double(), want[mine(r)].double())
                assert bool((m[:16 + o] == 9).all()) and bool((m[16 + o + count * es:] == 9).all())


@pytest.mark.parametrize("p", [1, 2])
def test_status_counts_operations(p):
    """Operations started and completed, on a communicator that has run nothing else and after an operation on staged kernels."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = H.Communicator.init_local(p, device=True, device_id=0)
    x, y = [torch.ones(1 << 12, device="cuda") for _ in range(p)], [torch.zeros(1 << 12, device="cuda") for _ in range(p)]
    for n in (1, 2, 3):
        c.all_reduce(x, y)
        assert c.sync() == 0
        st = c.status(p - 1)
        assert (st.head, st.tail) == (n, n) and "ops started %d, completed %d)" % (n, n) in c.describe_status(p - 1)
    c.all_reduce(x, y, nchan=2, algo=L.ALGO_MESH if p > 1 else L.ALGO_SINGLE)
    c.all_reduce(x, y)
    assert c.sync() == 0 and c.status(0).head == 5
    c.destroy()


@pytest.mark.parametrize("p", [1, 3])
def test_kernel_trace_is_filled(p, monkeypatch):
    """HCCL_KERNEL_TRACE at the communicator's creation: the selector's choice writes in-kernel timestamps."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    monkeypatch.setenv("HCCL_KERNEL_TRACE", "1")
    c = H.Communicator.init_local(p, device=True, device_id=0)
    x, y = [torch.ones(3 << 20, device="cuda") for _ in range(p)], [torch.zeros(3 << 20, device="cuda") for _ in range(p)]
    c.all_reduce(x, y)
    assert c.sync() == 0 and bool((y[0] == p).all())
    words = (C.c_uint64 * 16)()
    assert L.lib().HcclB200GetKernelTrace(c.handle, 0, words, 16, None) == 0
    assert 0 < words[0] < 2 ** 64 - 1 and any(words[1:])
    c.all_reduce(x, y, algo=L.ALGO_LOCAL)
    assert c.sync() == 0 and bool((y[p - 1] == p).all())
    c.destroy()


def test_select_names_what_runs(comms):
    """The selector's answer without a run: the direct kernels on ranks of one process, the single-rank copy for a lone rank."""
    c = comms(4)
    x, y = [torch.ones(1 << 18, device="cuda") for _ in range(4)], [torch.zeros(1 << 20, device="cuda") for _ in range(4)]
    c.all_reduce(x, [t[:1 << 18] for t in y])
    done(c, c.select(L.ALLREDUCE, 1 << 18, L.FP32)[0])
    c.all_gather(x, y)
    done(c, c.select(L.ALLGATHER, 1 << 18, L.FP32)[0])
    times = [c.select(L.ALLREDUCE, n, L.FP32)[2] for n in (1 << 10, 1 << 20, 1 << 24)]
    assert 0 < times[0] < times[1] < times[2]
    one = comms(1)
    one.all_reduce(x[:1], [y[0][:1 << 18]])
    done(one, one.select(L.ALLREDUCE, 1 << 18, L.FP32)[0])


@pytest.mark.parametrize("p", [2, 8])
@pytest.mark.parametrize("dtype", [torch.int8, torch.bfloat16, torch.float64])
@pytest.mark.parametrize("n", [1, 127, 129, 2048, 37_889, 75_777, 606_209])
def test_outputs_of_different_alignments(comms, p, dtype, n):
    """One element after the other: one per thread, a few CTAs more or less than two per SM, and as many as a tile of vectors holds."""
    c = comms(p)
    ins = rnd(p, n, dtype, n)
    base = [torch.full((n + 40,), 9, device="cuda", dtype=dtype) for _ in range(p)]
    outs = [b[8 + r:8 + r + n] for r, b in enumerate(base)]
    c.all_reduce(ins, outs, op=L.MAX)
    done(c)
    want = reduced(ins, L.MAX)
    for r, (b, o) in enumerate(zip(base, outs)):
        assert torch.equal(o.to(want.dtype), want)
        assert bool((b[:8 + r] == 9).all()) and bool((b[8 + r + n:] == 9).all())


@pytest.mark.parametrize("shift", [0, 4, 8, 1])
def test_large_copies(comms, shift):
    """More than 20 MB: a thread's full 128 bytes per tile.  Sources at the outputs' alignment, 16 bytes off it, and elsewhere; the
    size is no multiple of anything."""
    p, n = 3, 6_100_003
    c = comms(p)
    base = [torch.full((n + 40,), float(r), device="cuda") for r in range(p)]
    base[1].copy_(torch.arange(n + 40, device="cuda") % 16_777_213)
    bufs = [b[8 + (shift if r == 1 else 0):][:n] for r, b in enumerate(base)]
    want = bufs[1].clone()
    c.broadcast(bufs, 1)
    done(c)
    for r, (b, x) in enumerate(zip(base, bufs)):
        assert torch.equal(x, want)
        if r != 1:
            assert bool((b[:8] == r).all()) and bool((b[8 + n:] == r).all())


@pytest.mark.parametrize("p,root", [(2, 1), (5, 2)])
def test_rooted_and_variable_in_place(comms, p, root):
    c = comms(p)
    n = 50_021
    big = rnd(p, n * p, torch.float32, 1)
    want = [big[root][r * n:(r + 1) * n].clone() for r in range(p)]
    outs = [big[r][r * n:(r + 1) * n] for r in range(p)]
    c.scatter(big, outs, root)                                   # the root's own block stays where it is
    done(c)
    assert all(torch.equal(o, w) for o, w in zip(outs, want))
    full = rnd(p, n * p, torch.float32, 2)
    ins = [full[r][r * n:(r + 1) * n] for r in range(p)]
    want = torch.cat(ins)
    c.gather(ins, full, root)
    done(c)
    assert torch.equal(full[root], want)
    bufs = rnd(p, n, torch.float32, 3)
    want = reduced(bufs, L.SUM)
    c.reduce(bufs, bufs, root)
    done(c)
    check(bufs[root], want, torch.float32, p)
    counts = np.array([1000 + 37 * r for r in range(p)], np.uint64)
    displs = np.array([5 + 1500 * r for r in range(p)], np.uint64)
    cut = lambda x, r: x[int(displs[r]):int(displs[r] + counts[r])]
    full = rnd(p, n, torch.float32, 4)
    want = [cut(full[r], r).clone() for r in range(p)]
    c.all_gather_v([cut(full[r], r) for r in range(p)], full, counts, displs)
    done(c)
    assert all(torch.equal(cut(f, r), want[r]) for f in full for r in range(p))
    ins = rnd(p, n, torch.float32, 5)
    want = reduced(ins, L.SUM)
    c.reduce_scatter_v(ins, [cut(ins[r], r) for r in range(p)], counts, displs)
    done(c)
    for r in range(p):
        check(cut(ins[r], r), cut(want, r), torch.float32, p)
