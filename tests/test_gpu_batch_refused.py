"""A ray batch on a stream that is being captured is refused (it waits for its stream), for as often as one likes, and
the batches behind it are right: in both BVH formats, few rays and many."""
import ctypes

import numpy as np
import pytest

import pathtracer
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bvh", [pathtracer.BVH8_Q8, pathtracer.BVH2_FP32])
@pytest.mark.parametrize("n", [33, 60001])
def test_batches_behind_refused_ones(gpu_renderer, scene_factory, bvh, n):
    import torch
    s = scene_factory("spheres-10k")
    r = gpu_renderer
    r.upload_scene(s)
    rays = scenes.hit_ray_set(s, n, seed=n)
    tri, uvt = r.trace_closest_np(rays, bvh)
    d = torch.from_numpy(rays).cuda()
    t = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    u = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    cudart = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()
    for _ in range(20):   # more often than batches can be in flight
        assert cudart.cudaStreamBeginCapture(ctypes.c_void_p(stream.cuda_stream), 2) == 0   # relaxed
        with pytest.raises(pathtracer.GptError):
            r.intersect_closest(d, t, u, stream=stream.cuda_stream, bvh_format=bvh)
        graph = ctypes.c_void_p()
        assert cudart.cudaStreamEndCapture(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph)) != 0
        cudart.cudaGetLastError()
    torch.cuda.synchronize()
    assert bool((t == -7).all())
    for _ in range(2):
        t2, u2 = r.trace_closest_np(rays, bvh)
        assert np.array_equal(t2, tri) and np.array_equal(u2.view(np.uint32), uvt.view(np.uint32))
