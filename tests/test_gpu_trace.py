"""Traversal parity: GPU closest / any hit vs the CPU oracle (brute force and
its own binary BVH).  Hits are bit-exact: same canonical triangle id, same
t, beta, gamma bits, for every ray (the closest-hit rule is the minimum of
(t, id), which does not depend on the tree)."""
import numpy as np
import pytest

from globillum_gb300 import scenes

pytestmark = pytest.mark.gpu


def _oracle(sc, use_bvh):
    from oracle import oracle
    return oracle.OracleScene(sc, use_bvh=use_bvh)


def _check_closest(g, o):
    assert np.array_equal(g["ref"], o["ref"]), f"{(g['ref'] != o['ref']).sum()} triangle ids differ"
    hit = o["ref"] != 0xFFFFFFFF
    for k in ("t", "beta", "gamma"):
        assert np.array_equal(g[k][hit].view(np.uint32), o[k][hit].view(np.uint32)), k


@pytest.mark.parametrize("use_bvh", [False, True])
def test_cornell_closest_any(gpu_ctx, use_bvh):
    sc = scenes.cornell()
    scene = gpu_ctx.scene(sc)
    orc = _oracle(sc, use_bvh)
    o, d = scenes.random_rays(sc, 50000, seed=3)
    tmax = np.full(o.shape[0], 3.4e38, np.float32)
    _check_closest(scene.trace_closest(o, d, tmax), orc.trace_closest(o, d, tmax))
    tmax2 = np.random.default_rng(4).uniform(0.0, 1.5, o.shape[0]).astype(np.float32)
    _check_closest(scene.trace_closest(o, d, tmax2), orc.trace_closest(o, d, tmax2))
    assert np.array_equal(scene.trace_any(o, d, tmax2), orc.trace_any(o, d, tmax2))
    scene.close()


def test_icospheres_closest_any(gpu_ctx):
    sc = scenes.icospheres(n_spheres=40, level=3, box=20.0)
    scene = gpu_ctx.scene(sc)
    orc = _oracle(sc, True)
    o, d = scenes.random_rays(sc, 100000, seed=5)
    tmax = np.full(o.shape[0], 3.4e38, np.float32)
    g = scene.trace_closest(o, d, tmax)
    _check_closest(g, orc.trace_closest(o, d, tmax))
    assert (g["ref"] != 0xFFFFFFFF).mean() > 0.2
    tm = np.random.default_rng(6).uniform(0.0, 30.0, o.shape[0]).astype(np.float32)
    assert np.array_equal(scene.trace_any(o, d, tm), orc.trace_any(o, d, tm))
    scene.close()


def test_edge_rays(gpu_ctx):
    """Empty batch, negative max_t (no ray), axis-parallel directions, NaN
    rays and origins inside the room."""
    sc = scenes.cornell()
    scene = gpu_ctx.scene(sc)
    orc = _oracle(sc, False)
    empty = np.zeros((0, 3), np.float32)
    assert scene.trace_closest(empty, empty, np.zeros(0, np.float32)).shape == (0,)
    rng = np.random.default_rng(7)
    n = 6000
    o = rng.uniform(0.01, 0.99, size=(n, 3)).astype(np.float32)
    axes = np.eye(3, dtype=np.float32)
    d = np.concatenate([axes, -axes] * (n // 6))
    tmax = np.full(n, 3.4e38, np.float32)
    tmax[::7] = -1.0
    g = scene.trace_closest(o, d, tmax)
    _check_closest(g, orc.trace_closest(o, d, tmax))
    assert (g["ref"][::7] == 0xFFFFFFFF).all()
    # grid-aligned origins on the quad seams (x = 0.5 / z = 0.5 lines)
    o2 = o.copy()
    o2[:, 0] = 0.5
    o2[:, 2] = 0.5
    _check_closest(scene.trace_closest(o2, d, np.full(n, 3.4e38, np.float32)),
                   orc.trace_closest(o2, d, np.full(n, 3.4e38, np.float32)))
    bad = np.full((4, 3), np.nan, np.float32)
    h = scene.trace_closest(bad, bad, np.full(4, 1.0, np.float32))
    assert (h["ref"] == 0xFFFFFFFF).all()
    assert not scene.trace_any(bad, bad, np.full(4, 1.0, np.float32)).any()
    scene.close()


def _special_rays(sc, n):
    """Random rays, a sixteenth of them odd: negative, NaN, infinite and zero
    max_t, axis-parallel, zero and NaN directions, NaN and infinite origins."""
    o, d = scenes.random_rays(sc, n, seed=11)
    r = np.random.default_rng(12)
    t = np.where(r.uniform(size=n) < 0.5, 3.4e38, r.uniform(0.0, 40.0, n)).astype(np.float32)
    kind = r.integers(0, 128, n)
    for k, v in enumerate((-1.0, np.nan, np.inf, 0.0)):
        t[kind == k] = v
    d[kind == 4] = (0.0, 0.0, -1.0)
    d[kind == 5, 1] = 0.0
    d[kind == 6] = 0.0
    d[kind == 7, 0] = np.nan
    o[kind == 8, 2] = np.nan
    o[kind == 9, 0] = np.inf
    return o, d, t


@pytest.mark.parametrize("spheres", [1, 2, 3, 4, 19, 20])
def test_ray_counts(gpu_ctx, spheres):
    """Counts of rays around the lanes of the ray loop's grid (7 blocks of 128 on
    each SM), where its queue begins, and twice that, for trees on both
    sides of every line between the loop and a ray per lane; each call twice
    in a row, from host and from device memory.  All equal the oracle and, so,
    each other."""
    import ctypes as C

    import torch
    lanes = 7 * 128 * torch.cuda.get_device_properties(0).multi_processor_count
    sc = scenes.icospheres(n_spheres=spheres, level=3, box=12.0)
    top = 300007
    o, d, t = _special_rays(sc, top)
    orc = _oracle(sc, True)
    closest, occluded = orc.trace_closest(o, d, t), orc.trace_any(o, d, t)
    assert 0.05 < (closest["ref"] != 0xFFFFFFFF).mean() < 0.95
    s = gpu_ctx.scene(sc)
    lib, p = gpu_ctx.lib, C.c_void_p
    dev = [torch.from_numpy(x).cuda() for x in (o, d, t)]
    hits = torch.empty((top, 4), dtype=torch.float32, device="cuda")
    occl = torch.empty(top, dtype=torch.uint8, device="cuda")
    try:
        for n in (1, 31, 129, lanes - 1, lanes, lanes + 1, 2 * lanes, 2 * lanes + 1, top):
            for _ in range(2):
                _check_closest(s.trace_closest(o[:n], d[:n], t[:n]), closest[:n])
                assert np.array_equal(s.trace_any(o[:n], d[:n], t[:n]), occluded[:n])
            hits.zero_()
            occl.fill_(7)
            torch.cuda.synchronize()
            ptr = [p(x.data_ptr()) for x in dev]
            gpu_ctx.check(lib.gb_trace_closest(gpu_ctx.h, s.h, n, *ptr, p(hits.data_ptr()), 1))
            gpu_ctx.check(lib.gb_trace_any(gpu_ctx.h, s.h, n, *ptr, p(occl.data_ptr()), 1))
            g = hits.cpu().numpy()
            _check_closest({"t": g[:n, 0], "beta": g[:n, 1], "gamma": g[:n, 2], "ref": g[:n, 3].view(np.uint32)}, closest[:n])
            assert np.array_equal(occl.cpu().numpy()[:n], occluded[:n])
            assert (g[n:] == 0).all() and (occl.cpu().numpy()[n:] == 7).all()
    finally:
        s.close()
