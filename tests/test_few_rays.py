"""Ray batches of few rays (a warp per ray) and of more (a lane per ray) against the binary FP32 BVH, bit for bit: both
are conservative and ties go to the smaller input index."""
import numpy as np
import pytest

import pathtracer
import scenes


def ray_mix(scene, n):
    rays = scenes.hit_ray_set(scene, n, seed=n)
    rays[n // 2:, 7] = np.float32(3.0)      # segments
    rays[::5, 6] = np.float32(-2.0)         # hits behind the origin count
    rays[1::7, 6:8] = [[np.float32(2.0), np.float32(1.0)]]   # an empty interval
    rays[2::11, 3:6] = [[1.0, 0.0, 0.0]]
    return rays


# 9 resident blocks of 4 warps on each of 148 multiprocessors, 8 rays per warp: 42,624 is the last size of the first kind
@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 33, 5329, 21313, 42624, 42625])
@pytest.mark.parametrize("name", ["cornell", "cornell-all", "spheres-10k", "spheres-200k"])
def test_batches_equal_the_binary_bvh(gpu_renderer, scene_factory, name, n):
    s = scene_factory(name)
    rays = ray_mix(s, n)
    r = gpu_renderer
    r.upload_scene(s)
    tri, uvt = r.trace_closest_np(rays, pathtracer.BVH2_FP32)
    occ = r.trace_any_np(rays, pathtracer.BVH2_FP32)
    for build in (pathtracer.BVH_BUILD_HOST, pathtracer.BVH_BUILD_DEVICE):
        r.set_bvh_build(build)
        r.upload_scene(s)
        t8, u8 = r.trace_closest_np(rays)
        assert np.array_equal(t8, tri) and np.array_equal(u8.view(np.uint32), uvt.view(np.uint32))
        assert np.array_equal(r.trace_any_np(rays), occ)
    r.set_bvh_build(pathtracer.BVH_BUILD_HOST)


@pytest.mark.gpu
def test_batches_of_several_threads(gpu_renderer, scene_factory):
    """20 threads with streams of their own on one renderer (16 batches can be in flight) and batches of both kinds."""
    import threading
    import torch
    s = scene_factory("spheres-10k")
    r = gpu_renderer
    r.upload_scene(s)
    batches = []
    for n in (1, 700, 60001):
        rays = ray_mix(s, n)
        batches.append((torch.from_numpy(rays).cuda(),) + r.trace_closest_np(rays))
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for i in range(12):
                rays, tri, uvt = batches[(i + k) % 3]
                t = torch.empty(rays.shape[0], dtype=torch.int32, device="cuda")
                u = torch.empty((rays.shape[0], 3), dtype=torch.float32, device="cuda")
                r.intersect_closest(rays, t, u, stream=stream.cuda_stream)
                if not (np.array_equal(t.cpu().numpy().view(np.uint32), tri) and np.array_equal(u.cpu().numpy(), uvt)):
                    wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
