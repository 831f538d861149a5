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


def _fit_jobs(ctx, n, w=24, h=20):
    data = [scenes.cornell(width=w, height=h + k, spp=2, max_bounces=3, seed=k) for k in range(n)]
    for sc in data:
        sc.render["rng_mode"] = gbpt.GB_RNG_MRG32K3A_POOL
    hs = [ctx.scene(sc) for sc in data]
    jobs = [(s, sc.camera, sc.render) for s, sc in zip(hs, data)]
    return hs, jobs, [s.render(sc.camera, sc.render) for s, sc in zip(hs, data)]


def _loss(img, target):
    d = (img - target).astype(np.float64)  # float differences, squared and summed in double
    return float((d * d).sum())


@pytest.mark.parametrize("share", ["none", "own", "earlier", "later", "ring", "one image"])
def test_fit_images_that_share_memory(gpu_ctx, share):
    """A fitting step takes the scenes in their order: each loss reads its target
    as the images of the scenes before it have left it, and of images in the same
    place the last one stays.  Two steps, since a later scene's image is
    an earlier one's target only from the second step on.  A sum of 1,500 squares
    in double in another order differs by less than 1500 * 2^-53 of itself."""
    import torch
    hs, jobs, imgs = _fit_jobs(gpu_ctx, 3, h=20)
    n = [im.size for im in imgs]
    buf = torch.full((6, max(n)), 0.25, dtype=torch.float32, device="cuda")
    target, image = [0, 1, 2], [3, 4, 5]  # rows of buf
    if share == "own":
        image = target
    elif share == "earlier":
        target[1] = image[0]
    elif share == "later":
        target[0] = image[2]
    elif share == "ring":
        target = [image[2], image[0], image[1]]
    elif share == "one image":
        image = [3, 3, 3]
    try:
        gpu_ctx.fit_prepare(jobs, [buf[k].data_ptr() for k in target], [buf[k].data_ptr() for k in image])
        xs = [s.get_params() for s in hs]
        model = [np.full(max(n), 0.25, np.float32) for _ in range(6)]
        for step in range(2):
            _, loss = gpu_ctx.fit_step(xs)
            for k in range(3):
                want = _loss(imgs[k].reshape(-1), model[target[k]][: n[k]])
                assert abs(loss[k] - want) <= 1500 * 2.0 ** -53 * want, (step, k)
                model[image[k]][: n[k]] = imgs[k].reshape(-1)
            assert np.array_equal(buf.cpu().numpy(), np.stack(model)), step
    finally:
        for s in hs:
            s.close()


@pytest.mark.parametrize("offset", [0, 4, 2])
@pytest.mark.parametrize("managed", [False, True])
def test_fit_image_anywhere_in_an_allocation(gpu_ctx, memory, offset, managed):
    import torch
    hs, jobs, imgs = _fit_jobs(gpu_ctx, 1)
    target = torch.zeros(imgs[0].size, device="cuda")
    try:
        p = memory.device(imgs[0].nbytes + offset, managed)
        gpu_ctx.fit_prepare(jobs, [target.data_ptr()], [p + offset])
        gpu_ctx.fit_step([hs[0].get_params()])
        got = memory.read(p, imgs[0].nbytes + offset)
        assert np.array_equal(got[offset:], imgs[0].view(np.uint8).reshape(-1))
        assert (got[:offset] == 0xAB).all()
        short = memory.device(imgs[0].nbytes // 2)
        with pytest.raises(gbpt.GBError):
            gpu_ctx.fit_prepare(jobs, [target.data_ptr()], [short])
        assert (memory.read(short, imgs[0].nbytes // 2) == 0xAB).all()
    finally:
        for s in hs:
            s.close()
