"""The calls of csrc/python/fastcall.c through ctypes, for interpreters that it has not been and cannot be compiled for (no C
compiler or no Python headers): same functions, same refusals, several microseconds more per call."""
import ctypes as C

from . import _lib as L
from .utils.dtypes import data_ptr, numel


def _addresses(x, nlocal, needed=False):
    xs = [x] if nlocal == 1 and not isinstance(x, (list, tuple)) else x
    if len(xs) != nlocal:
        raise AssertionError("need one buffer per local rank")
    at = [data_ptr(b) for b in xs]
    if needed and not all(at):
        raise TypeError("every rank needs a buffer, got None or one without memory")
    return (C.c_void_p * nlocal)(*at)


def _layer(address):
    return C.cast(C.c_void_p(address), C.POINTER(L.MoeLayer))


class Calls:
    def __init__(self, lib):
        self._lib = lib

    def setup(self, dtypes, get_device, get_stream):
        self._dtypes, self._get_device, self._get_stream = dtypes, get_device, get_stream

    def op(self, comm, nlocal, coll, algo, nchan, op, root, send, recv, stream, by_recv, divide):
        of = recv if by_recv else send
        if nlocal > 1 or (isinstance(of, (list, tuple)) and of):
            of = of[0]
        if stream is None:
            stream = self._get_stream(self._get_device())
        return self.collective(comm, nlocal, coll, algo, nchan, self._dtypes[of.dtype], op, root, numel(of) // divide, send, recv, stream, None)

    def collective(self, comm, nlocal, coll, algo, nchan, dtype, op, root, count, send, recv, stream, tables):
        o = L.B200Op(coll=coll, algo=algo, nchan=nchan, dataType=dtype, op=op, root=root, count=count)
        names = () if tables is None else ("counts", "displs") if len(tables) == 2 else ("sendCounts", "sdispls", "recvCounts", "rdispls")
        for name, table in zip(names, tables or ()):
            setattr(o, name, table.ctypes.data)
        at = (None, None) if coll == L.BARRIER else (_addresses(send, nlocal), _addresses(recv, nlocal))
        return self._lib.HcclB200Collective(comm, C.byref(o), at[0], at[1], stream)

    def moe_dispatch(self, comm, nlocal, layer, x, topk_idx, stream):
        at = [_addresses(t, nlocal, True) for t in (x, topk_idx)]
        return self._lib.HcclB200MoeDispatchLocal(comm, _layer(layer), *at, stream)

    def moe_combine(self, comm, nlocal, layer, rows, topk_idx, gates, out, stream):
        at = [_addresses(t, nlocal, True) for t in (topk_idx, gates, out)]
        rows = C.cast(C.c_void_p(rows), C.POINTER(C.c_void_p)) if rows else None
        return self._lib.HcclB200MoeCombineLocal(comm, _layer(layer), rows, *at, stream)
