"""Diffuse textures with ray-differential mip selection (material.h:88-170,
hybrid-pt.cpp:300-328, material-cpu.cpp:36-77): GPU frames against the
oracle's restatement, fed the same MRG32k3a pools, bit for bit; textured and
plain scenes in one batch; direct lighting with textures; and the calls that
do not cover textures refusing them."""
import ctypes as C

import numpy as np
import pytest

from globillum_gb300 import gbpt, scenes

pytestmark = pytest.mark.gpu


def _pair(ctx, sc, rd):
    from oracle import oracle
    s = ctx.scene(sc)
    img = s.render(sc.camera, rd)
    s.close()
    n = rd["width"] * rd["height"]
    pool = ctx.mrg_pool(n, rd["spp"] * rd["max_bounces"], seed=rd.get("seed", 0))
    ref = oracle.OracleScene(sc, use_bvh=False).render(sc.camera, rd, pool)
    return img, ref


@pytest.mark.parametrize("rng_mode", [gbpt.GB_RNG_HALTON_LIGHT, gbpt.GB_RNG_MRG32K3A_POOL])
def test_textured_cornell_frame(gpu_ctx, rng_mode):
    sc = scenes.with_textures(scenes.cornell(width=64, height=48, spp=4, max_bounces=5), fraction=0.7, scale=2.0)
    rd = dict(sc.render, rng_mode=rng_mode)
    img, ref = _pair(gpu_ctx, sc, rd)
    assert np.array_equal(img, ref.astype(np.float32)), np.abs(img - ref).max()
    plain, _ = _pair(gpu_ctx, scenes.cornell(width=64, height=48, spp=4, max_bounces=5), rd)
    assert not np.array_equal(img, plain)


def test_textured_principled_icospheres_frame(gpu_ctx):
    base = scenes.icospheres(n_spheres=20, level=2, box=10.0, width=48, height=32, spp=3, max_bounces=4, n_lights=2)
    sc = scenes.with_textures(base, n_textures=3, size=32, fraction=0.6, scale=0.5, seed=5)
    assert any(m["principled"] >= 0 and m["diffuse_texture"] >= 0 for m in sc.materials)
    img, ref = _pair(gpu_ctx, sc, dict(sc.render))
    assert np.array_equal(img, ref.astype(np.float32)), np.abs(img - ref).max()


def test_textured_and_plain_scenes_in_one_batch(gpu_ctx):
    a = scenes.with_textures(scenes.cornell(width=40, height=32, spp=3, max_bounces=4), fraction=1.0, scale=3.0)
    b = scenes.cornell(width=24, height=24, spp=2, max_bounces=3, seed=2)
    sa, sb = gpu_ctx.scene(a), gpu_ctx.scene(b)
    single = [sa.render(a.camera, a.render), sb.render(b.camera, b.render)]
    for graph in (False, True):
        out = gpu_ctx.render_batch([(sa, a.camera, a.render), (sb, b.camera, b.render)], graph=graph)
        assert all(np.array_equal(x, y) for x, y in zip(out, single))
    sa.close()
    sb.close()


def test_textured_direct_lighting(gpu_ctx):
    from oracle import oracle
    sc = scenes.with_textures(scenes.cornell(width=48, height=40), fraction=1.0, scale=2.0)
    rd = dict(sc.render, shadow_offset=1e-3)
    s = gpu_ctx.scene(sc)
    img = s.render_direct(sc.camera, rd, 4)
    s.close()
    pool = gpu_ctx.mrg_pool(48 * 40, 3, seed=0)
    ref = oracle.OracleScene(sc, use_bvh=True).render_direct(sc.camera, rd, 4, pool)
    assert np.array_equal(img, ref)


def test_texture_errors(gpu_ctx):
    sc = scenes.with_textures(scenes.cornell(width=16, height=16, spp=1, max_bounces=2), fraction=1.0)
    bad = scenes.SceneData(**{**sc.__dict__, "materials": [dict(m, diffuse_texture=5) for m in sc.materials]})
    with pytest.raises(gbpt.GBError, match="texture index"):
        gpu_ctx.scene(bad)
    with pytest.raises(gbpt.GBError, match="texture coordinates"):
        gpu_ctx.scene(scenes.SceneData(**{**sc.__dict__, "texcoords": None}))
    tc = sc.texcoords.copy()
    tc[3, 1] = np.nan
    with pytest.raises(gbpt.GBError, match="non-finite texture"):
        gpu_ctx.scene(scenes.SceneData(**{**sc.__dict__, "texcoords": tc}))
    s = gpu_ctx.scene(sc)
    with pytest.raises(gbpt.GBError) as ei:
        s.backward(sc.camera, sc.render, np.ones((16, 16, 3), np.float32))
    assert ei.value.code == gbpt.GB_ERR_UNSUPPORTED
    cam, desc = gbpt.make_camera(sc.camera), gbpt.make_render_desc(sc.render)
    rc = gpu_ctx.lib.gb_render_noalloc(s.h, C.byref(cam), C.byref(desc), C.c_void_p(16), None)
    assert rc == gbpt.GB_ERR_UNSUPPORTED
    s.close()


@pytest.mark.parametrize("seed", [0, 1])
def test_colours_of_textured_materials(gpu_ctx, seed):
    """x^2.2 of a textured material's colours on the device (float pairs, with
    doubles to decide) against the oracle's doubles: a wall of 256 x 64 cells of
    a material each under a white texture, colours of every size from 2^-30 to 2^30,
    zero, one, and the ends of the range of the float pairs."""
    from oracle import oracle
    w, h = 256, 64
    r = np.random.default_rng(seed)
    n = w * h
    colour = np.exp2(r.uniform(-30.0, 30.0, (n, 3))).astype(np.float32)
    colour[: n // 2] = r.uniform(0.0, 1.0, (n // 2, 3)).astype(np.float32)
    ends = np.array([2.0 ** -20, 2.0 ** 20, 0.0, 1.0, 0.5, 1e-38], np.float32)
    edge = np.concatenate([ends, np.nextafter(ends, np.float32(0)), np.nextafter(ends, np.float32(np.inf))])
    colour.reshape(-1)[r.integers(0, 3 * n, 6000)] = edge[r.integers(0, edge.size, 6000)]
    x, y = np.meshgrid(np.arange(w + 1.0), np.arange(h + 1.0))
    p = np.stack([x / w * 4.0 - 2.0, y / h - 0.5, np.zeros_like(x)], -1)  # 4 x 1 at z = 0, seen from z = -2
    a, b, c, d = p[:-1, :-1], p[:-1, 1:], p[1:, 1:], p[1:, :-1]
    tri = np.stack([np.stack([a, b, c], 2), np.stack([a, c, d], 2)], 2).reshape(2 * n, 3, 3)
    tc = np.stack([tri[..., 0] * 0.1 + 0.5, tri[..., 1] * 0.1 + 0.5], -1)
    base = scenes.cornell()
    params = [dict(color=tuple(map(float, k)), roughness=0.6, metallic=float(m), specular=0.5)
              for k, m in zip(colour, r.choice([0.0, 0.5, 1.0], n))]
    sc = scenes.SceneData(
        tri.reshape(2 * n, 9).astype(np.float32), np.tile(np.float32([0, 0, -1]), (2 * n, 3)),
        np.repeat(np.arange(n), 2).astype(np.int32),
        [{"diffuse": (0.5, 0.5, 0.5), "principled": i, "diffuse_texture": 0} for i in range(n)], params,
        [dict(base.lights[0], center=(0.0, 0.0, -3.0), dir=(0.0, 0.0, 1.0), up=(0.0, 1.0, 0.0), wh=(1.0, 1.0))],
        dict(base.camera, pos=(0.0, 0.0, -2.0), dir=(0.0, 0.0, 1.0), up=(0.0, 1.0, 0.0), fovy_deg=27.0, aperture=0.0),
        dict(base.render, width=2 * w, height=2 * h, spp=2, max_bounces=1, rng_mode=gbpt.GB_RNG_MRG32K3A_POOL, ray_offset=1e-3,
             shadow_offset=1e-3),
        textures=[np.full((64, 64, 4), 255, np.uint8)], texcoords=tc.reshape(2 * n, 6).astype(np.float32))
    s = gpu_ctx.scene(sc)
    img = s.render(sc.camera, sc.render)
    s.close()
    pool = gpu_ctx.mrg_pool(4 * n, 2)
    ref = oracle.OracleScene(sc, use_bvh=True).render(sc.camera, sc.render, pool).astype(np.float32)
    assert len(np.unique(ref)) > 0.4 * ref.size  # most pixels show a colour of their own
    assert np.array_equal(img, ref, equal_nan=True)
