"""Result arrays come from the pool of the context they are made for, and from plain
memory when it has none to give."""
import ctypes as C
import gc

import numpy as np

from rabbitbin_b200 import api


class _Lib:
    def __init__(self, give):
        self.give, self.asked, self.freed, self.blocks = give, [], [], {}

    def rbg_result_alloc_on(self, handle, nbytes):
        self.asked.append((handle, nbytes))
        if not self.give:
            return None
        b = C.create_string_buffer(nbytes)
        self.blocks[C.addressof(b)] = b
        return C.addressof(b)

    def rbg_result_free(self, addr):
        self.freed.append(addr)


class _Ctx:
    def __init__(self, give):
        self._L, self._h = _Lib(give), object()


def test_pool_of_the_context():
    ctx = _Ctx(True)
    a = api._result(ctx, (1024, 512), np.float32)
    assert ctx._L.asked == [(ctx._h, 2 << 20)] and a.ctypes.data in ctx._L.blocks
    a[...] = 3.0
    view, addr = a[5:], a.ctypes.data
    del a
    gc.collect()
    assert ctx._L.freed == [] and view[0, 0] == 3.0
    del view
    gc.collect()
    assert ctx._L.freed == [addr]


def test_plain_memory_otherwise():
    ctx = _Ctx(False)
    a = api._result(ctx, (1024, 512), np.float32)
    assert len(ctx._L.asked) == 1 and a.shape == (1024, 512) and not a.any()
    small = api._result(_Ctx(True), (16, 16), np.uint32)
    assert small.flags.owndata
