"""BVH8 child blocks: header origins and scales over the coordinate range, leaves of several triangles.

Hits of the BVH8 equal those of the binary FP32 BVH bit for bit (the queries are conservative and ties go to the
smaller input index), so the comparisons need no tolerance."""
import numpy as np
import pytest

import pathtracer
import scenes


def transformed(name, scale, offset):
    s = scenes.config_scene(name)
    positions = (s.positions.astype(np.float64) * scale + np.asarray(offset, dtype=np.float64)).astype(np.float32)
    return scenes.Scene(positions, s.normals, s.tangents, s.uvs, s.material_ids, s.materials, camera=s.camera)


# coordinates around zero, far from it on either side (the origin's grid is then coarser than the boxes), tiny and
# huge; at 1e-30 box areas underflow, so the host builder's depth limit leaves leaves of several triangles
TRANSFORMS = [(1.0, (0, 0, 0)), (1.0, (-10, -5, -10)), (1.0, (1e5, -1e5, 3e4)), (1.0, (-1e6, 0, 1e6)), (1e-12, (0, 0, 0)),
              (1e-30, (0, 0, 0)), (1e10, (0, 0, 0)), (1e-3, (0, 50, 0))]


@pytest.mark.parametrize("scale,offset", TRANSFORMS)
@pytest.mark.parametrize("name", ["cornell-all", "spheres-10k"])
def test_host_built_blocks_contain_their_subtrees(name, scale, offset):
    r = pathtracer.bvh8_check(transformed(name, scale, offset))
    assert r["violations"] == 0 and r["misplaced"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("scale,offset", TRANSFORMS)
@pytest.mark.parametrize("name", ["cornell-all", "spheres-10k"])
def test_block_traversal_equals_the_binary_bvh(gpu_renderer, name, scale, offset):
    s = transformed(name, scale, offset)
    rays = scenes.hit_ray_set(scenes.config_scene(name), 20011)
    # scaled rays: origins and lengths follow the scene, directions stay unit vectors
    rays[:, 0:3] = rays[:, 0:3] * np.float32(scale) + np.asarray(offset, dtype=np.float32)
    rays[:, 6] = np.float32(1e-4 * scale)
    # axis-parallel rays: their clamped reciprocals overflow in the slab tests of large scenes
    axis = rays[:3001].copy()
    axis[:, 3:6] = np.repeat(np.concatenate([np.eye(3), -np.eye(3)]), 501, 0)[:3001].astype(np.float32)
    rays = np.concatenate([rays, axis])
    r = gpu_renderer
    r.upload_scene(s)
    tri, uvt = r.trace_closest_np(rays, pathtracer.BVH2_FP32)
    occ = r.trace_any_np(rays, pathtracer.BVH2_FP32)
    builds = [pathtracer.BVH_BUILD_HOST] + ([pathtracer.BVH_BUILD_DEVICE] if scale > 1e-30 else [])
    for build in builds:
        r.set_bvh_build(build)
        r.upload_scene(s)
        check = r.check_bvh(s)
        assert check["containment_violations"] == 0 and check["triangles_not_exactly_once"] == 0
        assert check["leaf_triangles"] == s.triangle_count
        t8, u8 = r.trace_closest_np(rays)
        assert np.array_equal(t8, tri) and np.array_equal(u8.view(np.uint32), uvt.view(np.uint32))
        assert np.array_equal(r.trace_any_np(rays), occ)
    r.set_bvh_build(pathtracer.BVH_BUILD_HOST)


@pytest.mark.gpu
def test_leaves_of_several_triangles_in_packed_scenes():
    # the second scene holds a cluster of triangles whose box areas underflow, so some of its leaves have several
    # triangles; its blocks (with those triangles behind them) are rebased behind the first scene's
    room, tiny = scenes.config_scene("cornell-all"), transformed("spheres-10k", 1e-30, (0, 0, 0))
    n = tiny.triangle_count
    s = scenes.Scene(np.concatenate([room.positions, tiny.positions]),
                     np.concatenate([room.normals, tiny.normals]), np.concatenate([room.tangents, tiny.tangents]),
                     np.concatenate([room.uvs, tiny.uvs]), np.concatenate([room.material_ids, np.zeros(n, np.uint32)]),
                     room.materials, camera=room.camera)
    assert pathtracer.bvh8_check(s)["misplaced"] == 0
    w, h, spp, depth = 48, 32, 4, 6
    cam = scenes.scene_camera(room, w, h)
    srv = pathtracer.Server(0, pool_size=1 << 18, variant="det")
    frame = pathtracer.Renderer(0, variant="det")
    try:
        srv.add_scene(scenes.config_scene("cornell"))
        job = srv.submit(srv.add_scene(s), cam, w, h, spp, depth)
        srv.wait(job)
        image, _ = srv.result(job)
        # the cluster's triangles are too small to be hit: the frame is the room's
        for scene in (s, room):
            frame.upload_scene(scene)
            frame.render_frame(cam, w, h, spp, depth, True)
            assert np.array_equal(frame.framebuffer(), image)
    finally:
        srv.close()
        frame.close()
