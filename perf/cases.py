"""Performance cases of the path tracer: what a program that uses it has it do, through its public binding.

Each case is a dict of plain values. Kinds:
  closest, any   ray batches on device memory (picking, probes, visibility and occlusion queries)
  frame          one rendered frame with its RGBA8 image and its float accumulation
  batch          several jobs over resident scenes through the job server, images read back
  upload         a changed scene uploaded with the device BVH build, then queried
  lights         a light alias table built on the device without allocating

Scenes are the repository's own named workloads; the camera, the sample streams, the rays, the scene's
vertices (upload) and the light weights come from the seed. The geometry of a named scene is an asset
that a program loads once, so it is generated once per process.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "gpu-path-tracer_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import pathtracer  # noqa: E402
import scenes  # noqa: E402
import workloads  # noqa: E402

# Knobs that gpt_autotune picks for frames of many pool-fulls of samples; a program tunes once and keeps them.
TUNED = dict(pool_size=1 << 24, trace_occupancy=10, trace_refill=16 | (4 << 8), trace_block=128)
TRIANGLES = {"cornell": 36, "cornell-all": 38, "cornell-textured": 38, "spheres-10k": 10258, "spheres-50k": 51234,
             "spheres-100k": 102434, "spheres-200k": 204866, "spheres-500k": 512130, "spheres-1m": 1310978,
             "spheres-2m": 2048258}
FIELDS = ("spheres-10k", "spheres-50k", "spheres-100k", "spheres-200k", "spheres-500k", "spheres-1m", "spheres-2m")
ROOMS = ("cornell", "cornell-all", "cornell-textured")


def _frame(name, scene, width, height, spp, depth, **more):
    case = dict(name=name, kind="frame", scene=scene, width=width, height=height, spp=spp, depth=depth, nee=True,
                tuned=False, device_bvh=False, pcg=False, power=False, variant="product")
    case.update(more)
    return case


def listed():
    return [
        # picking or a few probes: the smallest call, all latency
        dict(name="pick-1k", kind="closest", scene="spheres-10k", rays=1023),
        # an ordinary query batch (baking, distance probes), half coherent and half incoherent rays
        dict(name="closest-262k", kind="closest", scene="spheres-200k", rays=262147),
        # a large visibility batch on the headline scene
        dict(name="any-2m", kind="any", scene="spheres-1m", rays=2097153),
        # rebuilding the light sampler of the largest benchmark scene's emitters (4,096) between frames
        dict(name="lights-4096", kind="lights", lights=4096),
        # deforming geometry: a million triangles uploaded again and queried
        dict(name="upload-1m", kind="upload", scene="spheres-1m", rays=65536),
        # interactive preview: one sample per pixel with default settings
        _frame("preview-640x360", "spheres-200k", 640, 360, 1, 8),
        # the Cornell benchmark frame with default settings
        _frame("cornell-512", "cornell", 512, 512, 16, 8),
        # image textures and all six shading models, odd size, without next-event estimation
        _frame("textured-333x217", "cornell-textured", 333, 217, 9, 12, nee=False),
        # the headline frame: 1.31M triangles, 1920x1080, 64 spp, depth 12
        _frame("frame-1m-64spp", "spheres-1m", 1920, 1080, 64, 12, tuned=True),
        # a 4K frame of a larger scene in the production modes (PCG32 streams, power-weighted lights, device BVH)
        _frame("frame-2m-4k", "spheres-2m", 3840, 2160, 4, 10, tuned=True, device_bvh=True, pcg=True, power=True),
        # a small render farm: uneven jobs over three resident scenes through the job server
        dict(name="batch-12", kind="batch", jobs=12, largest=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("closest", "any", "frame", "frame", "frame", "batch", "upload", "lights"))
    if kind in ("closest", "any"):
        return dict(kind=kind, scene=rng.choice(ROOMS + FIELDS), rays=_log_int(rng, 1, 2000000) | 1)
    if kind == "lights":
        return dict(kind=kind, lights=_log_int(rng, 1, 4096))
    if kind == "upload":
        return dict(kind=kind, scene=rng.choice(FIELDS[:-1]), rays=_log_int(rng, 1, 65536))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(1, 12), largest=_log_int(rng, 128, 1024))
    spp = rng.choice((1, 4, 9, 16, 25, 64))
    height = _log_int(rng, 16, min(2160, int(math.sqrt(1.3e8 / 1.8 / spp))))
    width = max(1, int(height * rng.uniform(0.6, 2.2)))
    width = min(width, int(1.3e8 / spp / height))
    field = rng.random() < 0.65
    case = _frame("", rng.choice(FIELDS if field else ROOMS), width, height, spp, rng.randint(2, 16),
                  nee=rng.random() < 0.75, tuned=width * height * spp > (1 << 23), device_bvh=rng.random() < 0.4,
                  pcg=rng.random() < 0.25, power=rng.random() < 0.25,
                  variant="det" if rng.random() < 0.2 else "product")
    del case["name"]
    return case


@functools.lru_cache(maxsize=None)
def _scene(name):
    return scenes.config_scene(name)


def _camera(scene, width, height, rng):
    """The scene's own camera, moved a little by the seed."""
    c = scene.camera
    size = float(np.linalg.norm(np.asarray(c["look_at"]) - np.asarray(c["position"])))
    position = np.asarray(c["position"]) + rng.uniform(-0.02, 0.02, 3) * size
    return scenes.make_camera(tuple(position), c["look_at"], c["fov_y"], width / height)


def _rays(scene, count, seed):
    return scenes.hit_ray_set(scene, count, seed=seed)


def _moved(scene, seed):
    """The scene with its vertices stretched by a few percent, as an animation frame would hold it."""
    rng = np.random.default_rng(seed)
    factor = rng.uniform(0.97, 1.03, 3).astype(np.float32)
    return scenes.Scene(scene.positions * factor, scene.normals, scene.tangents, scene.uvs, scene.material_ids,
                        scene.materials, name=scene.name, camera=scene.camera)


def _batch_jobs(case, seed):
    """Jobs of the batched mix: log-uniform resolution, 1 to 64 spp, depth 8 to 12; cameras and streams from the seed."""
    sizes = np.random.default_rng([case["jobs"], case["largest"]])
    rng = np.random.default_rng(seed)
    jobs = []
    for k in range(case["jobs"]):
        w, h = workloads.log_uniform_resolution(sizes, (64, 64), (case["largest"], case["largest"] * 9 // 16))
        spp = (1, 4, 16, 64)[k % 4]
        jobs.append(dict(scene=k % 3, width=w, height=h, spp=spp, depth=int(sizes.integers(8, 13)),
                         camera=workloads.orbit_camera(rng, w, h), rng_offset=int(rng.integers(0, 1 << 20))))
    return jobs


BATCH_SCENES = ("spheres-10k", "spheres-200k", "spheres-500k")


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "lights":
        # emitter areas of the benchmark scenes: triangles with a log-spread of sizes
        w = (0.5 * 10.0 ** rng.uniform(-1.0, 0.5, case["lights"])).astype(np.float32)
        weights = torch.from_numpy(w).cuda()
        return dict(kind=kind, weights=weights, bins=torch.empty((case["lights"], 4), dtype=torch.int32, device="cuda"))
    if kind == "batch":
        server = pathtracer.Server(0, pool_size=1 << 22)
        ids = [server.add_scene(_scene(name)) for name in BATCH_SCENES]
        return dict(kind=kind, server=server, ids=ids, jobs=_batch_jobs(case, seed))
    scene = _scene(case["scene"])
    renderer = pathtracer.Renderer(0, variant=case.get("variant", "product"))
    if kind == "frame":
        renderer.set_bvh_build(pathtracer.BVH_BUILD_DEVICE if case["device_bvh"] else pathtracer.BVH_BUILD_HOST)
        renderer.upload_scene(scene)
        width, height = case["width"], case["height"]
        renderer.init_rendering_buffers(width, height)
        settings = dict(rng_offset=int(rng.integers(0, 1 << 30)),
                        rng_policy=pathtracer.RNG_PCG32 if case["pcg"] else pathtracer.RNG_PHILOX,
                        light_sampling=pathtracer.LIGHTS_POWER if case["power"] else pathtracer.LIGHTS_AREA)
        if case["tuned"]:
            settings.update(TUNED)
        return dict(kind=kind, renderer=renderer, camera=_camera(scene, width, height, rng), width=width, height=height,
                    spp=case["spp"], depth=case["depth"], nee=case["nee"], settings=settings,
                    accumulation=torch.empty((width * height, 4), dtype=torch.float32, device="cuda"))
    n = case["rays"]
    state = dict(kind=kind, renderer=renderer)
    if kind == "upload":
        renderer.set_bvh_build(pathtracer.BVH_BUILD_DEVICE)
        scene = state["scene"] = _moved(scene, seed)
    else:
        renderer.upload_scene(scene)
    state["rays"] = torch.from_numpy(_rays(scene, n, seed)).cuda()
    if kind == "any":
        state["occluded"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    else:
        state["tri"] = torch.empty(n, dtype=torch.int32, device="cuda")
        state["uvt"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "lights":
        status = pathtracer.build_alias_table_noalloc(state["weights"], state["bins"])
        if status != 0:
            raise RuntimeError(f"alias table: status {status}")
        return dict(bins=state["bins"])
    if kind == "batch":
        server = state["server"]
        jobs = [server.submit(state["ids"][j["scene"]], j["camera"], j["width"], j["height"], j["spp"], j["depth"], True,
                              rng_offset=j["rng_offset"], keep_accumulation=True) for j in state["jobs"]]
        images = []
        for job in jobs:
            server.wait(job)
            images.append(server.result(job, accumulation=True))
            server.release(job)
        return dict(images=images)
    renderer = state["renderer"]
    if kind == "frame":
        renderer.render_frame(state["camera"], state["width"], state["height"], state["spp"], state["depth"], state["nee"],
                              **state["settings"])
        renderer.copy_accumulation_to(state["accumulation"])
        return dict(image=renderer.framebuffer(), accumulation=state["accumulation"])
    if kind == "any":
        renderer.intersect_any(state["rays"], state["occluded"])
        return dict(occluded=state["occluded"])
    if kind == "upload":
        renderer.upload_scene(state["scene"])
    renderer.intersect_closest(state["rays"], state["tri"], state["uvt"])
    out = dict(tri=state["tri"], uvt=state["uvt"])
    if kind == "upload":
        out["lights"] = renderer.alias_table()
        out["lights_power"] = renderer.alias_table(power=True)
    return out


def work(case):
    """Bytes: every input of the call read once (the scene's triangles with their attributes where they are shaded, the
    rays) and every output written once. Operations: a ray is narrowed down to its triangle through log8(triangles)
    levels of 8 boxes (6 multiply-adds, 6 comparisons each) and 3 triangle tests of 50; a path has about 2.6 rays
    (1.9 closest, 0.7 shadow) of 400 shading operations."""
    kind = case["kind"]
    if kind == "lights":
        return dict(bytes=20.0 * case["lights"], flops=8.0 * case["lights"])

    def ray_flops(triangles):
        return 8 * 18 * max(1.0, math.log(triangles, 8)) + 150

    if kind == "batch":
        pixels = flops = 0
        for j in _batch_jobs(case, 0):
            pixels += j["width"] * j["height"]
            paths = j["width"] * j["height"] * j["spp"]
            flops += paths * 2.6 * (ray_flops(TRIANGLES[BATCH_SCENES[j["scene"]]]) + 400)
        return dict(bytes=180.0 * sum(TRIANGLES[n] for n in BATCH_SCENES) + 20.0 * pixels, flops=float(flops))
    triangles = TRIANGLES[case["scene"]]
    if kind == "frame":
        pixels = case["width"] * case["height"]
        reached = min(triangles, 8 * pixels * case["spp"])
        return dict(bytes=180.0 * reached + 20.0 * pixels, flops=pixels * case["spp"] * 2.6 * (ray_flops(triangles) + 400))
    rays = case["rays"]
    out = 1 if kind == "any" else 16
    # only the triangles that some ray can reach have to be read
    bytes_in = 36.0 * min(triangles, 3 * rays) + 32.0 * rays
    if kind == "upload":
        # host arrays in (vertices, normals, tangents, uvs, material), records and tree out
        bytes_in = 148.0 * triangles * 2 + 32.0 * rays
        return dict(bytes=bytes_in + out * rays, flops=rays * ray_flops(triangles) + 300.0 * triangles)
    return dict(bytes=bytes_in + out * rays, flops=rays * ray_flops(triangles))


def exact(case, seed):
    """Closest hits (u, v, t) by testing every triangle in 64 bits. The other outputs have no 64-bit value: hit indices,
    occlusion bytes and images are whole numbers, and a path's radiance depends on discrete choices (lobes, roulette,
    lights) that its 32-bit random numbers and arithmetic make."""
    if case["kind"] not in ("closest", "upload") or TRIANGLES[case["scene"]] * case["rays"] > 1e11:
        return None
    scene = _scene(case["scene"])
    if case["kind"] == "upload":
        scene = _moved(scene, seed)
    p = torch.from_numpy(scene.positions).cuda().double()
    v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    normal = torch.linalg.cross(e1, e2)
    # every term of the test is a product of one 3- or 6-vector of the ray with one of the triangle, so the
    # tests of a chunk of rays are four matrix products: with m = o x d and n = e1 x e2,
    # det = -d.n, u det = e2.m + (v0 x e2).d, v det = -(e1.m + (v0 x e1).d), t det = o.n - v0.n
    by_u = torch.cat([e2, torch.linalg.cross(v0, e2)], 1).T.contiguous()
    by_v = -torch.cat([e1, torch.linalg.cross(v0, e1)], 1).T.contiguous()
    by_d = -normal.T.contiguous()
    offset = (v0 * normal).sum(1)
    rays = torch.from_numpy(_rays(scene, case["rays"], seed)).cuda().double()
    out = torch.zeros((case["rays"], 3), dtype=torch.float64, device="cuda")
    chunk = max(1, (1 << 28) // p.shape[0])
    for at in range(0, case["rays"], chunk):
        r = rays[at:at + chunk]
        o, d = r[:, 0:3], r[:, 3:6]
        md = torch.cat([torch.linalg.cross(o, d), d], 1)
        det = d @ by_d
        inverse = 1.0 / det
        u = (md @ by_u) * inverse
        v = (md @ by_v) * inverse
        t = (offset[None, :] + o @ by_d) * -inverse
        hit = (det.abs() >= 1e-7) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= r[:, 6:7]) & (t < r[:, 7:8])
        t = torch.where(hit, t, math.inf)
        best, index = t.min(1)
        some = torch.isfinite(best)
        rows = torch.nonzero(some)[:, 0]
        index = index[rows]
        out[at + rows] = torch.stack([u[rows, index], v[rows, index], best[rows]], 1)
    return dict(uvt=out)
