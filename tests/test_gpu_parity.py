"""GPU parity: the CUDA path through the C ABI against the CPU oracle.

Bar: visibility (triangle id per pixel), depth and the shadow map are
bit-exact; the RGBA8 sRGB colour is within 1/255 per channel.
"""
import numpy as np
import pytest

from kat_scenes import flat_scene, one_surface_per_triangle
from rosy_gb300 import scene as sc
from rosy_gb300.graphics import Graphics, render_scene

COLOR_TOL = 1  # 1/255 per channel


def check_parity(s, ref, out, color_tol=COLOR_TOL):
    assert np.array_equal(out["ids"], ref["ids"]), f"ids differ at {np.count_nonzero(out['ids'] != ref['ids'])} pixels"
    assert np.array_equal(out["depth"].view(np.uint32), ref["depth"].view(np.uint32)), "depth differs"
    assert np.array_equal(out["shadow"].view(np.uint32), ref["shadow"].view(np.uint32)), \
        f"shadow map differs at {np.count_nonzero(out['shadow'] != ref['shadow'])} texels"
    d = np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32))
    assert d.max() <= color_tol, f"colour differs by {d.max()} at {np.count_nonzero(d > color_tol)} channels"


def run(s, oracle):
    ref = oracle.render(s)
    out = render_scene(s)
    return ref, out


def variants():
    v = {}
    v["tiny_s0"] = lambda: sc.tiny(0)
    v["tiny_s1"] = lambda: sc.tiny(1)
    v["random_triangles_640x360"] = lambda: sc.random_triangles()
    v["random_triangles_s7_odd_size"] = lambda: sc.random_triangles(seed=7, triangles=1000, width=333, height=217,
                                                                    shadow_size=300, texture_size=128)

    def inside():  # camera inside the cube: near-plane and guard-band clipping
        s = sc.random_triangles(seed=3, triangles=2000, width=320, height=200, shadow_size=256, texture_size=64)
        view = sc.camera_look_at_origin((0.2, 0.1, 0.3))
        proj = sc.projection(320 / 200, np.radians(90.0))
        s.scene = sc.scene_record(view, proj, s.scene["sun_position"][0], np.eye(4), (0.2, 0.1, 0.3), 320, 200)
        s.scene["shadow_projection_near"] = s.cameras[0]["shadow_projection_near"]
        return s
    v["camera_inside_clipping"] = inside

    def nocull():
        s = sc.random_triangles(seed=4, triangles=800, width=256, height=256, shadow_size=256, texture_size=64)
        s.draw_config["cull_enabled"] = 0
        return s
    v["cull_disabled"] = nocull

    def reverse():
        s = sc.random_triangles(seed=5, triangles=800, width=256, height=144, shadow_size=256, texture_size=64)
        s.draw_config["reverse_winding_order_enabled"] = 1
        return s
    v["reverse_winding"] = reverse

    def pcf3():
        s = sc.random_triangles(seed=6, triangles=800, width=256, height=144, shadow_size=512, texture_size=64,
                                pcf_mode=sc.PCF_3X3)
        return s
    v["pcf_3x3"] = pcf3

    def nobias():
        s = sc.random_triangles(seed=8, triangles=800, width=256, height=144, shadow_size=512, texture_size=64)
        s.draw_config["depth_bias_enabled"] = 0
        return s
    v["bias_disabled"] = nobias

    def lambert():
        s = sc.random_triangles(seed=9, triangles=800, width=256, height=144, shadow_size=512, texture_size=64)
        s.scene["brdf_lighting_enabled"] = 0
        return s
    v["lambert"] = lambert

    def small_scene():
        return sc.scene_scale(seed=1, meshes=8, triangles_per_mesh=512, materials=4, texture_size=64, width=320,
                              height=180, shadow_size=512, frames=2)
    v["scene_scale_small"] = small_scene

    def world_space():
        s = sc.scene_scale(seed=2, meshes=6, triangles_per_mesh=512, materials=3, texture_size=64, width=320,
                           height=180, shadow_size=512, frames=2)
        s.scene["tangent_space_enabled"] = 0
        s.scene["ensure_orthogonal_bitangent"] = 1
        s.scene["flip_tangents"] = (1, 0, 1, 0)
        s.scene["flip_lights"] = (0, 1, 0, 1)
        return s
    v["world_space_flips"] = world_space

    v["blended_random_triangles"] = lambda: sc.with_blended(
        sc.random_triangles(seed=12, triangles=600, width=256, height=160, shadow_size=256, texture_size=64), 0.5)
    v["blended_scene_scale"] = lambda: sc.with_blended(
        sc.scene_scale(seed=5, meshes=6, triangles_per_mesh=512, materials=3, texture_size=64, width=320, height=180,
                       shadow_size=512, frames=1), 0.3, alpha=0.45)
    v["alpha_mask"] = lambda: sc.with_blended(
        sc.random_triangles(seed=13, triangles=400, width=200, height=120, shadow_size=256, texture_size=32), 0.5,
        alpha=1.0, mask_cutoff=0.5)
    def cascades(n, seed):
        def make():
            s = sc.random_triangles(seed=seed, triangles=800, width=256, height=160, shadow_size=256,
                                    texture_size=64)
            s.scene = s.scene.copy()
            P = s.scene["shadow_projection_near"][0].reshape(4, 4).copy()  # rows of the column-major array = columns
            P[:, 0:2] *= 16.0  # light extent 36 / 16 units: the cube spans several cascades
            s.scene["shadow_projection_near"] = P.reshape(1, 16)
            s.cameras = [s.scene]
            s.draw_config["shadow_cascades"] = n
            return s
        return make
    v["cascades_4"] = cascades(4, 14)
    v["cascades_2"] = cascades(2, 15)
    return v


VARIANTS = variants()


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(VARIANTS))
def test_parity(gpu, oracle, name):
    s = VARIANTS[name]()
    ref, out = run(s, oracle)
    assert (ref["ids"] > 0).any()
    check_parity(s, ref, out)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", list(range(16)))
def test_fragment_output_modes(gpu, oracle, mode):
    s = sc.scene_scale(seed=3, meshes=4, triangles_per_mesh=512, materials=2, texture_size=32, width=160,
                       height=96, shadow_size=256, frames=1)
    s.scene["fragment_output"] = mode
    ref, out = run(s, oracle)
    check_parity(s, ref, out)


@pytest.mark.gpu
def test_kat_scenes_on_gpu(gpu, oracle):
    a, b, c, d = (1.5, 1.5, 0.5), (5.5, 1.5, 0.5), (5.5, 5.5, 0.5), (1.5, 5.5, 0.5)
    t = ((0.0, 0.0, 0.4), (8.0, 0.0, 0.4), (0.0, 8.0, 0.4))
    for s in (flat_scene([(a, b, c), (a, c, d)]), one_surface_per_triangle(flat_scene([t, t, t])),
              flat_scene([((0.0, 0.0, 1.5), (8.0, 0.0, 0.5), (0.0, 8.0, 0.5))])):
        ref, out = run(s, oracle)
        check_parity(s, ref, out)


@pytest.mark.gpu
def test_frames_along_spline_reuse_context(gpu, oracle):
    """One context, several frames with new scene constants (graph replay)."""
    from rosy_gb300.graphics import Graphics

    s = sc.scene_scale(seed=4, meshes=8, triangles_per_mesh=512, materials=4, texture_size=64, width=320,
                       height=180, shadow_size=512, frames=4)
    g = Graphics()
    g.init(s.width, s.height, s.shadow_size)
    try:
        g.set_asset(s)
        g.set_graphic_objects(s.objects, s.surfaces)
        g.set_draw_config(s.draw_config)
        for i in range(4):
            si = s.with_camera(i)
            g.update(si.scene)
            g.render()
            g.sync()
            out = g.download()
            check_parity(si, oracle.render(si), out)
    finally:
        g.deinit()


@pytest.mark.gpu
def test_parity_scene_scale_full_size(gpu, oracle):
    """The bench workload itself (262,144 triangles, 1920x1080, 4096^2 shadow map,
    32 materials x 3 textures of 1024^2): bit-exact visibility/depth/shadow, colour
    within 1/255, on the first and a later spline frame."""
    s = sc.scene_scale(seed=0)
    for cam in (0, 5):
        si = s.with_camera(cam)
        ref, out = run(si, oracle)
        assert (ref["ids"] > 0).mean() > 0.05
        check_parity(si, ref, out)


def _msaa_variants():
    v = {}
    v["msaa_random_triangles"] = lambda: sc.random_triangles(seed=31, triangles=800, width=256, height=160,
                                                             shadow_size=256, texture_size=64)
    v["msaa_scene_scale"] = lambda: sc.scene_scale(seed=3, meshes=8, triangles_per_mesh=512, materials=4,
                                                   texture_size=64, width=320, height=180, shadow_size=512, frames=1)
    v["msaa_blended"] = lambda: sc.with_blended(
        sc.random_triangles(seed=32, triangles=600, width=256, height=160, shadow_size=256, texture_size=64), 0.5)
    v["msaa_alpha_mask"] = lambda: sc.with_blended(
        sc.random_triangles(seed=33, triangles=400, width=200, height=120, shadow_size=256, texture_size=32), 0.5,
        alpha=1.0, mask_cutoff=0.5)
    return v


MSAA_VARIANTS = _msaa_variants()


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(MSAA_VARIANTS))
def test_msaa_parity(gpu, oracle, name):
    """4x multisampling (the reference's default, src/Engine/Graphics.cpp:5605-5607):
    triangle id and depth per sample bit-exact, the resolved colour within 1/255."""
    s = MSAA_VARIANTS[name]()
    s.samples = 4
    ref = oracle.render(s)
    out = render_scene(s)
    assert out["ids"].shape == ref["ids"].shape == (4, s.height, s.width)
    assert np.array_equal(out["ids"], ref["ids"]), f"ids differ at {np.count_nonzero(out['ids'] != ref['ids'])} samples"
    assert np.array_equal(out["vis_depth"].view(np.uint32), ref["depth"].view(np.uint32)), "sample depth differs"
    assert np.array_equal(out["depth"].view(np.uint32), ref["depth"][0].view(np.uint32)), "depth output differs"
    assert np.array_equal(out["shadow"].view(np.uint32), ref["shadow"].view(np.uint32))
    d = np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32))
    assert d.max() <= COLOR_TOL, f"colour differs by {d.max()} at {np.count_nonzero(d > COLOR_TOL)} channels"
    # some pixels really are partially covered (the resolve mixes)
    assert (np.ptp(out["ids"], axis=0) > 0).any()


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,triangles", [(16, 16, 20000), (17, 15, 20000), (33, 1, 3000), (1, 40, 3000),
                                                    (47, 31, 1), (64, 48, 300)])
def test_msaa_tiles_of_one_to_four_triangles(gpu, oracle, width, height, triangles):
    """Tiles whose list of (pixel, triangle) pairs is full (a triangle per sample), ragged or nearly empty."""
    s = sc.random_triangles(seed=41, triangles=triangles, width=width, height=height, shadow_size=128, texture_size=32)
    if triangles > 10000:  # triangles of a pixel or less: four of them in most pixels
        v = s.vertices[:, 0:3].reshape(-1, 3, 3)
        s.vertices[:, 0:3] = (v[:, :1] + (v - v[:, :1]) * np.float32(0.12)).reshape(-1, 3)
        s.draw_config["cull_enabled"] = 0
    s.samples = 4
    ref, out = run(s, oracle)
    if triangles > 10000:
        assert (np.ptp(out["ids"], axis=0) > 0).mean() > 0.5
    assert np.array_equal(out["ids"], ref["ids"])
    assert np.array_equal(out["vis_depth"].view(np.uint32), ref["depth"].view(np.uint32))
    assert np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("chunk_stamps,small_extent,spread", [(8, 1, 1.0), (256, 16, 0.3), (32, 8, 0.08), (32, 16, 0.02)])
def test_msaa_raster_parts(gpu, oracle, chunk_stamps, small_extent, spread):
    """The four launches of a multisampled camera raster share out small, medium and screen-sized
    records, boxes cut by the viewport among them: every sample's id and depth as the oracle's."""
    s = sc.random_triangles(seed=43, triangles=900, width=307, height=205, shadow_size=64, texture_size=32)
    v = s.vertices[:, 0:3].reshape(-1, 3, 3)
    s.vertices[:, 0:3] = (1.4 * v[:, :1] + (v - v[:, :1]) * np.float32(spread)).reshape(-1, 3)
    s.samples = 4
    ref = oracle.render(s)
    g = Graphics()
    g.init(s.width, s.height, s.shadow_size, samples=4)
    try:
        g.set_asset(s)
        g.set_graphic_objects(s.objects, s.surfaces)
        g.set_draw_config(s.draw_config)
        g.set_tuning(chunk_stamps, small_extent)
        g.update(s.scene)
        for timed in (False, True):  # side by side, then one after the other
            g.set_stage_timing(timed)
            g.render()
            if g.sync_code() == 14:
                g.render()
            g.sync()
            out = g.download()
            assert np.array_equal(out["ids"], ref["ids"])
            assert np.array_equal(out["vis_depth"].view(np.uint32), ref["depth"].view(np.uint32))
    finally:
        g.deinit()


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [[0, 1, 0, 0, 255, 256, 257, 0], [1] * 300, [511, 1, 0, 512, 2], [769]])
def test_draw_tables(gpu, oracle, lengths):
    """Draws of no, one, and about 256 triangles (the step of the draw tables), opaque and blended, of two
    meshes whose vertices also straddle the step."""
    tris = sum(lengths)
    a = sc.random_triangles(seed=59, triangles=2 * tris, width=160, height=96, shadow_size=128, texture_size=32)
    v, i = 3 * tris, np.arange(3 * tris, dtype=np.uint32)
    a.meshes = [(0, v, 0, v), (v, v, v, v)]
    a.indices = np.concatenate([i, i])
    blended = np.concatenate([a.materials, a.materials])
    blended["alpha_mode"][1], blended["base_color_factor"][1, 3] = 2, 0.5
    a.materials = blended
    surfs = np.zeros(2 * len(lengths), sc.SURFACE_DTYPE)
    for m in range(2):
        at = 0
        for k, n in enumerate(lengths):
            s = surfs[m * len(lengths) + k]
            s["mesh_index"], s["start_index"], s["index_count"] = m, 3 * at, 3 * n
            s["material_index"], s["blended"] = m, m
            at += n
    a.surfaces = surfs
    a.draw_config["shadow_cascades"] = 2
    check_parity(a, *run(a, oracle))


@pytest.mark.gpu
@pytest.mark.parametrize("chunk_stamps,small_extent", [(8, 1), (16, 4), (33, 2), (64, 1), (256, 16)])
@pytest.mark.parametrize("spread,fov", [(0.03, 60.0), (0.3, 60.0), (1.0, 60.0), (1.0, 1.5)])
def test_raster_chunks(gpu, oracle, chunk_stamps, small_extent, spread, fov):
    """Chunks of fewer and of more than 32 stamps, of records of one stamp (more records than are staged) to
    screen-sized ones, boxes cut by the viewport, and (narrow field of view) vertices far outside it."""
    s = sc.random_triangles(seed=53, triangles=1500, width=318, height=211, shadow_size=190, texture_size=32, fov_deg=fov)
    v = s.vertices[:, 0:3].reshape(-1, 3, 3)
    s.vertices[:, 0:3] = (v[:, :1] + (v - v[:, :1]) * np.float32(spread)).reshape(-1, 3)
    ref = oracle.render(s)
    g = Graphics()
    g.init(s.width, s.height, s.shadow_size)
    try:
        g.set_asset(s)
        g.set_graphic_objects(s.objects, s.surfaces)
        g.set_draw_config(s.draw_config)
        g.set_tuning(chunk_stamps, small_extent)
        g.update(s.scene)
        g.render()
        if g.sync_code() == 14:
            g.render()
        g.sync()
        check_parity(s, ref, g.download())
    finally:
        g.deinit()


@pytest.mark.gpu
@pytest.mark.parametrize("samples", [1, 4])
@pytest.mark.parametrize("width,height,triangles,spread,mask", [
    (48, 40, 24000, 0.05, False),  # over 8,192 records (a window of group boxes), hundreds to a tile
    (33, 17, 1500, 0.8, True),     # tens of fragments to a pixel, some discarded
    (16, 16, 31, 1.0, False),      # less than a group
    (64, 1, 33, 1.0, False)])
def test_blended_lists(gpu, oracle, samples, width, height, triangles, spread, mask):
    """Blended lists of less than a group to several windows of groups, and pixels of many rounds."""
    s = sc.random_triangles(seed=47, triangles=triangles, width=width, height=height, shadow_size=64, texture_size=32)
    v = s.vertices[:, 0:3].reshape(-1, 3, 3)
    s.vertices[:, 0:3] = (v[:, :1] + (v - v[:, :1]) * np.float32(spread)).reshape(-1, 3)
    s = sc.with_blended(s, 0.95, alpha=0.3, mask_cutoff=0.4 if mask else None)
    s.samples = samples
    ref, out = run(s, oracle)
    assert np.array_equal(out["ids"], ref["ids"])
    assert np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("samples", [1, 4])
@pytest.mark.parametrize("width,height,triangles,spread", [
    (200, 120, 600, 6.0),  # deep overdraw by triangles that cover blocks whole
    (33, 17, 300, 3.0),    # records of the smallest extent on the block grid, and below it
    (71, 45, 400, 40.0)])  # boxes cut on every side, blocks cut by the viewport
def test_hidden_stamps(gpu, oracle, samples, width, height, triangles, spread):
    """Stamps behind a block's depth are not drawn; of equal depths the later triangle stays."""
    s = sc.random_triangles(seed=61, triangles=triangles, width=width, height=height, shadow_size=64, texture_size=16)
    v = s.vertices[:, 0:3].reshape(-1, 3, 3)
    v = v[:, :1] + (v - v[:, :1]) * np.float32(spread)
    v[triangles // 2:] = v[:triangles - triangles // 2]  # the same triangles again
    s.vertices[:, 0:3] = v.reshape(-1, 3)
    s.samples = samples
    ref, out = run(s, oracle)
    assert np.array_equal(out["ids"], ref["ids"])
    assert np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("samples", [1, 4])
@pytest.mark.parametrize("width,height,triangles,spread", [
    (2300, 19, 80, 60.0),  # edges of more than 2,048 pixels do not fit 32 bits over a tile
    (40, 40, 700, 0.6),    # tiles with more records than are prepared at a time
    (300, 31, 513, 0.02)])  # most tiles empty; records of a pixel or less
def test_blended_edges(gpu, oracle, samples, width, height, triangles, spread):
    s = sc.random_triangles(seed=53, triangles=triangles, width=width, height=height, shadow_size=64, texture_size=32)
    v = s.vertices[:, 0:3].reshape(-1, 3, 3)
    s.vertices[:, 0:3] = (v[:, :1] + (v - v[:, :1]) * np.float32(spread)).reshape(-1, 3)
    s = sc.with_blended(s, 0.9, alpha=0.3)
    s.samples = samples
    ref, out = run(s, oracle)
    assert np.array_equal(out["ids"], ref["ids"])
    assert np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL


@pytest.mark.gpu
def test_shading_error_against_fp64_oracle(gpu, oracle):
    """The oracle also shades in float64; the GPU's 8-bit sRGB colour stays within
    1.5 levels of that (0.5 of it is the 8-bit rounding itself)."""
    s = sc.scene_scale(seed=4, meshes=8, triangles_per_mesh=512, materials=4, texture_size=64, width=320,
                       height=180, shadow_size=512, frames=1)
    ref = oracle.render(s, fp64=True)
    out = render_scene(s)
    err = np.abs(out["color"][..., :3].astype(np.float64) - ref["color_f64"][..., :3] * 255.0)
    assert err.max() <= 1.5, err.max()
    assert err.mean() < 0.3, err.mean()


@pytest.mark.gpu
@pytest.mark.parametrize("shadow,samples", [(64, 1), (2880, 1), (2896, 1), (2880, 4)])
def test_frames_in_a_row_around_32_mb_of_targets(gpu, oracle, shadow, samples):
    """Setup and raster start as the launch before them ends where the depth targets take at most
    32 MB: frames in a row, each other's leftovers in the targets, on both sides of that."""
    from rosy_gb300.graphics import Graphics

    s = sc.scene_scale(seed=5, meshes=6, triangles_per_mesh=256, materials=3, texture_size=32, width=97, height=65,
                       shadow_size=shadow, frames=4)
    s.samples = samples
    g = Graphics()
    g.init(s.width, s.height, s.shadow_size, samples=samples)
    try:
        g.set_asset(s)
        g.set_graphic_objects(s.objects, s.surfaces)
        g.set_draw_config(s.draw_config)
        for cam in (0, 1, 2, 3, 1):
            g.update(s.cameras[cam])
            g.render()
            if cam == 0 and g.sync_code() == 14:
                g.render()
        g.sync()
        s.scene = s.cameras[1]
        ref, out = oracle.render(s), g.download()
        assert np.array_equal(out["ids"], ref["ids"])
        assert np.array_equal(out["shadow"].view(np.uint32), ref["shadow"].view(np.uint32))
        assert np.abs(out["color"].astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL
    finally:
        g.deinit()


@pytest.mark.gpu
def test_read_back_with_frames_in_flight(gpu, oracle):
    """Frames read back through rz_read_frame while the next ones render (two
    host buffers, rz_read_sync before refilling one): every buffer holds its own
    frame's colour and depth."""
    import torch

    from rosy_gb300.graphics import Graphics

    s = sc.scene_scale(seed=7, meshes=8, triangles_per_mesh=512, materials=4, texture_size=64, width=320,
                       height=180, shadow_size=512, frames=5)
    g = Graphics()
    g.init(s.width, s.height, s.shadow_size)
    try:
        g.set_asset(s)
        g.set_graphic_objects(s.objects, s.surfaces)
        g.set_draw_config(s.draw_config)
        g.update(s.cameras[0])
        g.render()
        if g.sync_code() == 14:
            g.render()
        g.sync()
        bufs = [(torch.empty((s.height, s.width, 4), dtype=torch.uint8, pin_memory=True).numpy(),
                 torch.empty((s.height, s.width), dtype=torch.float32, pin_memory=True).numpy()) for _ in range(2)]
        got = []
        for i in range(5):
            if i >= 2:
                g.read_sync(1)
                got.append((i - 2, bufs[i % 2][0].copy(), bufs[i % 2][1].copy()))
            g.update(s.cameras[i])
            g.render()
            g.read_frame(*bufs[i % 2])
        g.sync()
        for i in (3, 4):
            got.append((i, bufs[i % 2][0].copy(), bufs[i % 2][1].copy()))
        for i, color, depth in got:
            ref = oracle.render(s.with_camera(i))
            assert np.array_equal(depth.view(np.uint32), ref["depth"].view(np.uint32)), i
            assert np.abs(color.astype(np.int32) - ref["color"].astype(np.int32)).max() <= COLOR_TOL, i
    finally:
        g.deinit()
