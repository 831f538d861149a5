"""Images in the caller's device memory: a kernel packs straight into memory
that it can write as whole floats; any other place is written by a copy, and
an allocation that ends before the image does is refused."""
import ctypes as C

import numpy as np
import pytest

from globillum_gb300 import gbpt, scenes

pytestmark = pytest.mark.gpu


class _Memory:
    """Allocations of the driver in the context the library runs in."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        self.held = []

    def _ck(self, rc):
        assert rc == 0, f"driver error {rc}"

    def device(self, n, managed=False):
        p = C.c_uint64()
        if managed:
            self._ck(self.cu.cuMemAllocManaged(C.byref(p), C.c_size_t(n), 1))
        else:
            self._ck(self.cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(n)))
        self.held.append(p)
        self._ck(self.cu.cuMemsetD8_v2(p, 0xAB, C.c_size_t(n)))
        return p.value

    def read(self, p, n):
        out = np.empty(n, np.uint8)
        self._ck(self.cu.cuMemcpyDtoH_v2(C.c_void_p(out.ctypes.data), C.c_uint64(p), C.c_size_t(n)))
        return out

    def free(self):
        for p in self.held:
            self._ck(self.cu.cuMemFree_v2(p))


@pytest.fixture
def memory(gpu_ctx):
    m = _Memory()
    yield m
    m.free()


def _room(w=64, h=48):
    sc = scenes.cornell(width=w, height=h, spp=2, max_bounces=3)
    return sc, 12 * w * h


@pytest.mark.parametrize("managed", [False, True])
@pytest.mark.parametrize("offset", [0, 4, 20, 2, 7])
def test_image_anywhere_in_an_allocation(gpu_ctx, memory, managed, offset):
    """Whole and odd byte addresses, up to the allocation's last byte."""
    sc, n = _room()
    s = gpu_ctx.scene(sc)
    try:
        ref = s.render(sc.camera, sc.render).view(np.uint8).reshape(-1)
        p = memory.device(n + offset, managed)
        s.render_device(sc.camera, sc.render, p + offset)
        got = memory.read(p, n + offset)
        assert np.array_equal(got[offset:], ref)
        assert (got[:offset] == 0xAB).all()
    finally:
        s.close()


@pytest.mark.parametrize("size,offset", [(18432, 0), (1 << 20, (1 << 20) - 4 * 64 * 48), (1 << 20, (1 << 20) - 4)])
def test_allocation_that_ends_before_the_image(gpu_ctx, memory, size, offset):
    """Refused with the frame intact: nothing is written, and the image can
    still be read into memory that holds it."""
    sc, n = _room()
    s = gpu_ctx.scene(sc)
    try:
        ref = s.render(sc.camera, sc.render)
        p = memory.device(size)
        with pytest.raises(gbpt.GBError):
            s.render_device(sc.camera, sc.render, p + offset)
        assert (memory.read(p, size) == 0xAB).all()
        out = np.empty_like(ref)
        gpu_ctx.check(gpu_ctx.lib.gb_render_read(gpu_ctx.h, C.c_void_p(out.ctypes.data), 0))
        assert np.array_equal(out, ref)
    finally:
        s.close()
