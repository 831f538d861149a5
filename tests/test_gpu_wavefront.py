"""The slot-pool loop (host-driven, graph = 1) and the kernels that follow whole
paths (k_paths for small chunks, k_finish for the last paths of a chunk's
graph, graph = 2) at the sizes where they can go wrong: path counts around a
warp, a block and the shading tile, pools far smaller than the frame,
one-bounce paths (every path ends with its light sample still pending), a
scene without lights, every lobe of the principled room, textures with a sky.
Frames and gradients equal those of the oracle / of the other driver."""
import numpy as np
import pytest

from globillum_gb300 import gbpt, scenes

pytestmark = pytest.mark.gpu


def _against_oracle(ctx, sc, rd):
    from oracle import oracle
    s = ctx.scene(sc)
    img = s.render(sc.camera, rd)
    st = ctx.stats()
    s.close()
    n = rd["width"] * rd["height"]
    pool = ctx.mrg_pool(n, rd["spp"] * rd["max_bounces"], seed=rd.get("seed", 0))
    ref = oracle.OracleScene(sc, use_bvh=False).render(sc.camera, rd, pool)
    assert np.array_equal(img, ref.astype(np.float32)), np.abs(img - ref).max()
    assert st["camera_rays"] == n * rd["spp"]
    return st


@pytest.mark.parametrize("w,h,spp,slots", [(1, 1, 1, 1), (31, 1, 1, 0), (127, 1, 1, 0), (43, 3, 1, 0), (16, 16, 3, 129),
                                           (33, 31, 5, 100), (64, 65, 2, 4097)])
@pytest.mark.parametrize("bounces", [1, 2, 7])
@pytest.mark.parametrize("graph", [1, 2])
def test_path_counts_and_pools(gpu_ctx, w, h, spp, slots, bounces, graph):
    sc = scenes.principled_room(width=w, height=h, spp=spp, max_bounces=bounces, rr_start=3)
    old = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(graph=graph)
        if slots:
            gpu_ctx.set_tuning(slots=slots)
        _against_oracle(gpu_ctx, sc, sc.render)
    finally:
        gpu_ctx.set_tuning(slots=old["slots"], graph=old["graph"])


@pytest.mark.parametrize("w,h,spp,slots", [(512, 384, 1, 0), (513, 384, 1, 0), (512, 512, 1, 0), (513, 512, 1, 0),
                                           (300, 310, 3, 5000), (257, 129, 16, 0),
                                           (681, 800, 1, 0), (681, 801, 1, 0), (1024, 1023, 1, 0)])
@pytest.mark.parametrize("kind", ["room", "textured"])
def test_finish_of_a_chunk(gpu_ctx, w, h, spp, slots, kind):
    """Chunks at and above the 3 * 2^16 paths of k_paths: the graph's loop leaves
    its last paths to k_finish; the host-driven loop does not.  And queues at
    and above one shading tile of 512 per block (7 blocks on 152 SMs).  Same
    frames, same ray counts."""
    if kind == "room":
        sc = scenes.principled_room(width=w, height=h, spp=spp, max_bounces=5, rr_start=1)
    else:
        sc = scenes.with_textures(scenes.icospheres(n_spheres=30, level=2, box=12.0, width=w, height=h, spp=spp,
                                                    max_bounces=4, n_lights=1), scale=0.2)
        sc.lights.append({"type": gbpt.GB_LIGHT_SKY, "map": scenes.procedural_sky(32, 16), "scale": 0.5,
                          "diameter": 30.0, "power": -1.0})
        sc.camera.update(aperture=0.2, focus_distance=8.0)
    s = gpu_ctx.scene(sc)
    old = gpu_ctx.get_tuning()
    out = []
    try:
        for graph in (1, 2):
            gpu_ctx.set_tuning(graph=graph, **({"slots": slots} if slots else {}))
            img = s.render(sc.camera, sc.render)
            st = gpu_ctx.stats()
            out.append((img, [st[k] for k in ("camera_rays", "extension_rays", "shadow_rays", "light_samples")]))
    finally:
        gpu_ctx.set_tuning(graph=old["graph"], slots=old["slots"])
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1] and out[0][1][0] == w * h * spp


def test_no_lights_and_dark_light(gpu_ctx):
    sc = scenes.cornell(width=40, height=30, spp=2, max_bounces=4)
    rd = dict(sc.render, rng_mode=gbpt.GB_RNG_MRG32K3A_POOL)
    dark = scenes.SceneData(**{**sc.__dict__, "lights": []})
    assert _against_oracle(gpu_ctx, dark, rd)["shadow_rays"] == 0
    # the light faces away from all but the ceiling above it: most light
    # samples are exactly zero and trace no shadow ray
    away = scenes.SceneData(**{**sc.__dict__, "lights": [dict(sc.lights[0], dir=(0.0, 1.0, 0.0))]})
    st = _against_oracle(gpu_ctx, away, rd)
    assert 0 < st["shadow_rays"] < st["light_samples"] // 2


@pytest.mark.parametrize("slots", [97, 1024])
def test_adjoint_pool_size_does_not_matter(gpu_ctx, slots):
    """The visibility of a vertex's light sample reaches its record one
    iteration after the vertex: the gradient with a small pool (paths restart
    many times on a slot) equals the one with every path in flight, up to the
    order of the float atomics (1e-5 of the largest entry)."""
    sc = scenes.principled_room(width=29, height=23, spp=4, max_bounces=5, rr_start=2)
    sc.materials[5] = dict(sc.materials[4])  # the adjoint room without glass
    s = gpu_ctx.scene(sc)
    g = np.random.default_rng(3).normal(size=(23, 29, 3)).astype(np.float32)
    ref = s.backward(sc.camera, sc.render, g)
    old = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(slots=slots)
        got = s.backward(sc.camera, sc.render, g)
    finally:
        gpu_ctx.set_tuning(slots=old["slots"])
    s.close()
    assert np.abs(ref).max() > 0
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("scale", [1e-4, 1.0, 3e7, 2e12])
def test_axis_parallel_and_scaled_rays(gpu_ctx, scale):
    """Node tests at the ends of their range: rays parallel to one or two axes
    (inverse directions of 2^80), tiny and huge scenes, rays starting on a
    node's plane; closest and any hits equal the oracle's brute force."""
    from oracle import oracle
    sc = scenes.icospheres(n_spheres=6, level=2, box=8.0, width=8, height=8, spp=1, max_bounces=1, n_lights=1)
    sc.positions = (sc.positions.astype(np.float64) * scale).astype(np.float32)
    rng = np.random.default_rng(5)
    n = 6000
    p = sc.positions.reshape(-1, 3)
    tgt = p[rng.integers(0, p.shape[0], n)].astype(np.float64)
    d = rng.normal(size=(n, 3))
    k = rng.integers(0, 3, n)
    r = np.arange(n)
    d[r[: n // 2], k[: n // 2]] = 0.0                      # parallel to a plane
    axis = np.zeros((n, 3))
    axis[r, k] = rng.choice([-1.0, 1.0], n)
    d[n // 2: 3 * n // 4] = axis[n // 2: 3 * n // 4]       # parallel to an axis
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = tgt - d * scale * rng.choice([0.0, 3.0, 40.0], n)[:, None]
    o[:, 0] += rng.normal(size=n) * scale * 1e-3
    o, d = o.astype(np.float32), d.astype(np.float32)
    t = np.where(rng.uniform(size=n) < 0.5, 3.4e38, 10.0 * scale).astype(np.float32)
    orc = oracle.OracleScene(sc, use_bvh=False)
    s = gpu_ctx.scene(sc)
    a, b = s.trace_closest(o, d, t), orc.trace_closest(o, d, t)
    assert np.array_equal(a["ref"], b["ref"])
    hit = b["ref"] != 0xFFFFFFFF
    assert hit.mean() > 0.2
    for f in ("t", "beta", "gamma"):
        assert np.array_equal(a[f][hit].view(np.uint32), b[f][hit].view(np.uint32))
    assert np.array_equal(s.trace_any(o, d, t) != 0, orc.trace_any(o, d, t) != 0)
    s.close()


@pytest.mark.parametrize("w,h", [(1, 1), (33, 31), (64, 3)])
@pytest.mark.parametrize("cams,lights", [(1, 8), (3, 9), (2, 17)])
@pytest.mark.parametrize("sky", [False, True])
def test_direct_light_sample_groups(gpu_ctx, w, h, cams, lights, sky):
    """Light-sample counts around the groups the direct integrators trace
    together, image sizes around a warp and a block, with and without a sky:
    bit-equal to the oracle, sample by sample."""
    from oracle import oracle
    sc = scenes.icospheres(n_spheres=12, level=2, box=8.0, width=w, height=h, n_lights=2)
    if sky:
        sc.lights.append({"type": gbpt.GB_LIGHT_SKY, "map": scenes.procedural_sky(16, 8), "scale": 0.3,
                          "diameter": 20.0, "power": -1.0})
    rd = dict(sc.render, shadow_offset=0.01, seed=2)
    s = gpu_ctx.scene(sc)
    orc = oracle.OracleScene(sc, use_bvh=True)
    pool = gpu_ctx.mrg_pool(w * h, cams * lights + 1, seed=2)
    assert np.array_equal(s.render_direct(sc.camera, rd, lights), orc.render_direct(sc.camera, rd, lights, pool))
    assert np.array_equal(s.render_hybrid_direct(sc.camera, rd, cams, lights),
                          orc.render_hybrid_direct(sc.camera, rd, cams, lights, pool))
    s.close()


@pytest.mark.parametrize("builder", ["host", "device"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 24, 25, 77])
def test_small_trees_under_every_policy(gpu_ctx, builder, n):
    """Trees of one node and of a few, with leaves of one to three triangles in
    any slot: the leaf bits of a node name the right triangles for the voting
    policy, the postponing ones (groups on the stack) and the cooperative one."""
    from oracle import oracle
    rng = np.random.default_rng(n)
    c = rng.uniform(-2, 2, (n, 1, 3))
    pos = (c + rng.uniform(-1, 1, (n, 3, 3))).astype(np.float32).reshape(n, 9)
    base = scenes.cornell(width=24, height=20, spp=2, max_bounces=3)
    sc = scenes.SceneData(pos, None, np.zeros(n, np.int32), base.materials, [],
                          [dict(base.lights[0], center=(0.0, 5.0, 0.0), wh=(2.0, 2.0))],
                          dict(base.camera, pos=(0.0, 0.0, -6.0)), dict(base.render, rng_mode=gbpt.GB_RNG_MRG32K3A_POOL))
    s = gpu_ctx.scene(sc, builder=builder)
    pool = gpu_ctx.mrg_pool(24 * 20, 2 * 3)
    ref = oracle.OracleScene(sc, use_bvh=False).render(sc.camera, sc.render, pool).astype(np.float32)
    old = gpu_ctx.get_tuning()
    try:
        for mode in (1, 2, 3, 4):
            for graph in (1, 2):
                gpu_ctx.set_tuning(tri_mode=mode, graph=graph)
                assert np.array_equal(s.render(sc.camera, sc.render), ref), (mode, graph)
    finally:
        gpu_ctx.set_tuning(tri_mode=old["tri_mode"], graph=old["graph"])
        s.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 65, 700, 5000])
@pytest.mark.parametrize("kind", ["soup", "grid", "far", "flat"])
def test_refit_small_and_odd_trees(gpu_ctx, n, kind):
    """Refits of trees of one leaf, one node and many levels: after a refit to
    the vertices it was built from a tree costs the same node visits
    (the nodes are the same; counted under the policy that tests pending
    triangles before each node, since with the others a ray's visits depend on
    the rays that share its warp); after a refit to others the hits
    are the oracle's, and moving back restores the costs."""
    from oracle import oracle
    rng = np.random.default_rng(n)
    c = rng.uniform(-4.0, 4.0, (n, 1, 3))
    p = (c + rng.uniform(-0.4, 0.4, (n, 3, 3))).astype(np.float32)
    q = (c[::-1] * 0.8 + rng.uniform(-0.6, 0.6, (n, 3, 3))).astype(np.float32)
    if kind == "grid":  # box sides that are whole multiples of the planes' steps
        p, q = np.round(p * 4) / 4, np.round(q * 2) / 2
    elif kind == "far":
        p, q = p + np.float32(3.0e4), q + np.float32(3.0e4)
    elif kind == "flat":
        p[..., 1] = q[..., 1] = 0.5
    p, q = (np.ascontiguousarray(v.reshape(n, 9), dtype=np.float32) for v in (p, q))
    base = scenes.cornell()
    desc = {**base.__dict__, "normals": None, "texcoords": None, "material_index": np.zeros(n, np.int32)}
    sp, sq = (scenes.SceneData(**{**desc, "positions": v}) for v in (p, q))
    cam = dict(base.camera)
    mid = p.reshape(-1, 3).mean(0)
    cam.update(pos=(float(mid[0]), float(mid[1]) + 2.0, float(mid[2]) + 11.0), dir=(0.0, -0.15, -1.0), up=(0.0, 1.0, 0.0))
    rd = {**base.render, "width": 24, "height": 20, "spp": 2, "max_bounces": 2}
    s = gpu_ctx.scene(sp, builder="device")

    def cost():
        s.render(cam, rd, instrumented=True)
        st = gpu_ctx.stats()
        return st["closest_node_visits"], st["shadow_node_visits"]

    old = gpu_ctx.get_tuning()["tri_mode"]
    gpu_ctx.set_tuning(tri_mode=4)
    try:
        built = cost()
        assert cost() == built
        s.refit(p)
        assert cost() == built
    finally:
        gpu_ctx.set_tuning(tri_mode=old)
    s.refit(q)
    o, d = scenes.random_rays(sq, 4000, seed=n)
    tmax = np.full(o.shape[0], 3.4e38, np.float32)
    got = s.trace_closest(o, d, tmax)
    ref = oracle.OracleScene(sq, use_bvh=False).trace_closest(o, d, tmax)
    assert np.array_equal(got["ref"], ref["ref"])
    hit = ref["ref"] != 0xFFFFFFFF
    for k in ("t", "beta", "gamma"):
        assert np.array_equal(got[k][hit].view(np.uint32), ref[k][hit].view(np.uint32)), k
    s.refit(p)
    gpu_ctx.set_tuning(tri_mode=4)
    try:
        assert cost() == built
    finally:
        gpu_ctx.set_tuning(tri_mode=old)
        s.close()


@pytest.mark.parametrize("wa,wb", [(40, 7), (5000, 4728), (5001, 4728), (20000, 28640), (20001, 28640)])
@pytest.mark.parametrize("spp", [1, 9])
def test_paths_per_warp(gpu_ctx, wa, wb, spp):
    """Chunks whose warps follow 8, 16 or 32 paths, at the edges between them
    (8 * 1216 and 16 * 3040 paths) and, with more samples, for the last paths of
    larger chunks: lanes without a path trace for a path of another scene.
    Same images and ray counts as the host-driven loop."""
    sa = scenes.principled_room(width=wa, height=1, spp=spp, max_bounces=5, rr_start=1)
    sb = scenes.with_textures(scenes.icospheres(n_spheres=30, level=2, box=12.0, width=wb, height=1, spp=spp,
                                                max_bounces=4, n_lights=2), scale=0.2)
    handles = [gpu_ctx.scene(sa), gpu_ctx.scene(sb)]
    jobs = [(h, sc.camera, sc.render) for h, sc in zip(handles, (sa, sb))]
    out = []
    try:
        for graph in (False, True):
            imgs = gpu_ctx.render_batch(jobs, graph=graph)
            st = gpu_ctx.stats()
            out.append((imgs, [st[k] for k in ("camera_rays", "extension_rays", "shadow_rays", "light_samples")]))
    finally:
        for h in handles:
            h.close()
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    assert out[0][1] == out[1][1] and out[0][1][0] == (wa + wb) * spp


def test_fit_step_after_a_frame_of_another_layout(gpu_ctx):
    """A fitting step after a render that used the same buffers for other
    pixels: the step's frame is again that of the batch, whatever the other
    frame left in them."""
    import torch
    big = scenes.cornell(width=160, height=120, spp=4, max_bounces=3)
    big.render["seed"] = 5
    small = scenes.principled_room(width=24, height=20, spp=2, max_bounces=3)
    small.render["rng_mode"] = gbpt.GB_RNG_MRG32K3A_POOL
    hb, hs = gpu_ctx.scene(big), gpu_ctx.scene(small)
    try:
        hb.render(big.camera, big.render)  # the buffers are large enough for both from here on
        x = hs.get_params()
        target = torch.zeros(20, 24, 3, device="cuda")
        image = torch.empty_like(target)
        gpu_ctx.fit_prepare([(hs, small.camera, small.render)], [target.data_ptr()], [image.data_ptr()])
        gpu_ctx.fit_step([x])
        first = image.cpu().numpy()
        hb.render(big.camera, big.render)
        gpu_ctx.fit_step([x])
        assert np.array_equal(image.cpu().numpy(), first)
        assert np.array_equal(hs.render(small.camera, small.render), first)
    finally:
        hb.close()
        hs.close()


@pytest.mark.parametrize("other", [(40, 30, 0), (40, 30, 3), (30, 40, 0), (64, 48, 0)])
def test_light_draws_of_a_layout_are_kept(gpu_ctx, other):
    """Frames with Halton and with MRG32k3a light draws in turns: of one layout
    they need no other launches than the same frame again does, and of several
    (another seed, size or order of sizes) every frame stays the same."""
    w, h, seed = other
    a = scenes.cornell(width=40, height=30, spp=2, max_bounces=4)
    s = gpu_ctx.scene(a)
    halton, mrg = (dict(a.render, rng_mode=m) for m in (gbpt.GB_RNG_HALTON_LIGHT, gbpt.GB_RNG_MRG32K3A_POOL))
    mixed = dict(a.render, width=w, height=h, seed=seed, rng_mode=gbpt.GB_RNG_HALTON_LIGHT)

    def render(rd):
        img = s.render(a.camera, rd)
        return img, gpu_ctx.stats()["kernel_launches"]

    try:
        ref = []
        for rd in (halton, mrg, mixed):
            render(rd)
            ref.append(render(rd))
        render(halton)
        for _ in range(2):  # one layout: nothing is started anew
            for rd, (img, n) in ((mrg, ref[1]), (halton, ref[0])):
                got, m = render(rd)
                assert np.array_equal(got, img) and m == n
        for rd, k in ((mixed, 2), (mrg, 1), (halton, 0), (mixed, 2), (halton, 0), (mrg, 1)):
            assert np.array_equal(render(rd)[0], ref[k][0])
    finally:
        s.close()


@pytest.mark.parametrize("fit_mode,view_mode", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_fit_steps_between_views(gpu_ctx, fit_mode, view_mode):
    """Fitting steps with a view of another layout between them: the step keeps
    its graph (it allocates nothing, so an allocation set to fail does not
    matter) and its frames, losses and the view stay what they were."""
    import torch
    a = scenes.principled_room(width=24, height=20, spp=2, max_bounces=3)
    b = scenes.cornell(width=31, height=9, spp=3, max_bounces=2, seed=4)
    for sc in (a, b):
        sc.render["rng_mode"] = fit_mode
    hs = [gpu_ctx.scene(sc) for sc in (a, b)]
    view = dict(a.render, width=33, height=17, spp=1, rng_mode=view_mode, seed=9)
    lib = gpu_ctx.lib
    try:
        targets = [torch.zeros(20, 24, 3, device="cuda"), torch.zeros(9, 31, 3, device="cuda")]
        images = [torch.empty_like(t) for t in targets]
        xs = [h.get_params() for h in hs]
        seen = hs[0].render(a.camera, view)
        gpu_ctx.fit_prepare([(h, sc.camera, sc.render) for h, sc in zip(hs, (a, b))],
                            [t.data_ptr() for t in targets], [t.data_ptr() for t in images])
        _, loss = gpu_ctx.fit_step(xs)
        first = [t.cpu().numpy() for t in images]
        for h, sc, im in zip(hs, (a, b), first):
            assert np.array_equal(h.render(sc.camera, sc.render), im)
        gpu_ctx.fit_step(xs)
        for _ in range(2):
            assert np.array_equal(hs[0].render(a.camera, view), seen)
            for t in images:
                t.zero_()
            torch.cuda.synchronize()
            lib.gb_set_fault_injection(0)
            try:
                _, again = gpu_ctx.fit_step(xs)
            finally:
                lib.gb_set_fault_injection(-1)
            assert np.array_equal(again, loss)
            for t, im in zip(images, first):
                assert np.array_equal(t.cpu().numpy(), im)
    finally:
        for h in hs:
            h.close()


@pytest.mark.parametrize("materials", [6, 3000])
def test_gradient_copies(gpu_ctx, materials):
    """A float sum of the gradient holds the terms of one block of the adjoint,
    however many parameters there are.  Terms of 2^-27 are lost where they follow
    one of 1 in the same sum: 152 large pixels among 2^18, in tiles of 128 that
    760 blocks (5 on each SM) take two or three of each, can lose the terms of at
    most 152 * 3 tiles of 2048, 22 % (25 % with the spread of the terms' sizes);
    a fifth of the sums loses about twice as much."""
    sc = scenes.cornell(width=512, height=512, spp=1, max_bounces=1)
    sc.render["rng_mode"] = gbpt.GB_RNG_MRG32K3A_POOL
    sc.materials += [dict(sc.materials[0]) for _ in range(materials - len(sc.materials))]
    s = gpu_ctx.scene(sc)
    img = s.render(sc.camera, sc.render)[..., 1].reshape(-1)
    lit = np.flatnonzero((img > np.median(img[img > 0])) & (img < 0.99))
    big = np.random.default_rng(1).choice(lit, 152, replace=False)
    small = np.full(512 * 512, 2.0 ** -27, np.float32)
    small[big] = 0.0
    large = np.zeros(512 * 512, np.float32)
    large[big] = 1.0

    def light_gradient(g):  # the light's green emission
        full = s.backward(sc.camera, sc.render, np.repeat(g[:, None], 3, 1).reshape(512, 512, 3))
        return float(full[5 * len(sc.materials) + 1])

    try:
        a, b, both = light_gradient(small), light_gradient(large), light_gradient(small + large)
        assert a > 0 and b > 100 * a
        lost = (a + b - both) / a
        print("lost", lost)
        assert -0.02 < lost < 0.25
    finally:
        s.close()


def _three_scenes():
    """A room with Halton light draws, a textured soup under a sky through a lens,
    and a plain soup with two lights: 200x150 at 7 spp, 300x250 at 5 and
    31x23 at 6."""
    room = scenes.principled_room(width=200, height=150, spp=7, max_bounces=5, rr_start=2)
    soup = scenes.with_textures(scenes.icospheres(n_spheres=30, level=2, box=12.0, width=300, height=250, spp=5,
                                                  max_bounces=4, n_lights=1), scale=0.2)
    soup.lights.append({"type": gbpt.GB_LIGHT_SKY, "map": scenes.procedural_sky(32, 16), "scale": 0.5, "diameter": 30.0,
                        "power": -1.0})
    soup.camera.update(aperture=0.2, focus_distance=8.0)
    plain = scenes.icospheres(n_spheres=9, level=2, box=9.0, width=31, height=23, spp=6, max_bounces=6, n_lights=2)
    return [room, soup, plain]


@pytest.fixture(scope="module")
def three_references(gpu_ctx):
    from oracle import oracle
    out = []
    for sc in _three_scenes():
        rd = sc.render
        pool = gpu_ctx.mrg_pool(rd["width"] * rd["height"], rd["spp"] * rd["max_bounces"], seed=rd.get("seed", 0))
        out.append(oracle.OracleScene(sc, use_bvh=True).render(sc.camera, rd, pool).astype(np.float32))
    return out


@pytest.mark.parametrize("sample_mb,slots,graph", [(1024, 4099, True), (1024, 4099, False), (4, 4099, True), (4, 1 << 24, True),
                                                   (4, 70000, True), (4, 70000, False), (2, 333, True), (2, 333, False)])
def test_large_frames_with_small_pools(gpu_ctx, three_references, sample_mb, slots, graph):
    """Frames beyond the chunks that follow whole paths, with pools far smaller
    than they are: paths restart on used slots inside the captured loop (textured,
    under a sky, through a lens, of several scenes), k_finish takes what is
    left, and chunks of both kinds follow one another (4 MB of samples: two
    rounds of 105,713 pixels through the loop, the last 167,000 paths whole).
    Every image equals the oracle's."""
    data = _three_scenes()
    hs = [gpu_ctx.scene(sc) for sc in data]
    old = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(slots=slots, sample_mb=sample_mb)
        got = gpu_ctx.render_batch([(h, sc.camera, sc.render) for h, sc in zip(hs, data)], graph=graph)
        for g, ref in zip(got, three_references):
            assert np.array_equal(g, ref), np.abs(g - ref).max()
        st = gpu_ctx.stats()
        assert st["camera_rays"] == sum(sc.render["width"] * sc.render["height"] * sc.render["spp"] for sc in data)
        for h, sc, ref in zip(hs[:2], data, three_references):
            gpu_ctx.set_tuning(graph=2 if graph else 1)
            assert np.array_equal(h.render(sc.camera, sc.render), ref)
    finally:
        gpu_ctx.set_tuning(slots=old["slots"], sample_mb=old["sample_mb"], graph=old["graph"])
        for h in hs:
            h.close()
