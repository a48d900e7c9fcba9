"""The workloads whose speed matters, each through the framework's public entry points.

Frames come from a seeded room scene (kinectfusion_b200.synthetic) rendered on
the GPU at any image size; volumes cover the room's 5.12 m cube unless a case
says otherwise.  Kinds of case:

  track    a new sequence tracked and fused frame by frame, then the model
           rendered at the last pose: host depth frames, two in flight
           (PipelinedReconstruction) or one at a time (Reconstruction.process)
  batch    several sequences of different resolution stepped together, frames
           in device memory, then each model rendered
  fuse     frames with known poses (another tracker, a turntable, a robot):
           pyramid and integration per frame, then one render
  render   the surface maps of a mapped volume at one pose, into device memory
  pyramid  the depth pyramid of one frame
  icp      a level of Gauss-Newton steps against given model maps, or (steps
           0) one sweep of the normal equations, as a host-side solver asks for
  mesh     the triangle mesh of a mapped volume, in host memory
  train    optimiser steps of the learned warm start, then its weights

Outputs that a 64-bit restatement can be given for have one in `exact`.
Everything behind a TSDF update or a ray march has none: which pixel a voxel
reads, which samples a ray takes and where it stops are decided by 32-bit
rounding, so a 64-bit rerun is another volume and another image.
"""

import ctypes as C
import math

import numpy as np
import torch

import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, learned, synthetic
from kinectfusion_b200.pipeline import PipelinedReconstruction, lib
from kinectfusion_b200.pipeline_set import DeviceSurfaceMaps

VOXELS = {"float": abi.KF_VOXEL_FLOAT, "int16": abi.KF_VOXEL_QUANTIZED, "bf16": abi.KF_VOXEL_BF16}
RULES = {"angle": abi.KF_RULE_ANGLE_WEIGHTED, "classic": abi.KF_RULE_CLASSIC}


# ---- the cases --------------------------------------------------------------------------
def _volume(res, voxel="float", color=False, rule="angle", sparse=False, band=False, res_y=0, res_z=0):
    return {"res": res, "res_y": res_y or res, "res_z": res_z or res, "voxel_m": 5.12 / res, "voxel": voxel,
            "color": color, "rule": rule, "sparse": sparse, "band": band or sparse, "all_corners": False,
            "cell_normals": False}


def listed():
    return [
        # a whole 30-frame pass of the headline workload: 640x480 into 512^3 float voxels of 1 cm
        {"name": "track_512", "kind": "track", "width": 640, "height": 480, "frames": 30, "in_flight": 2,
         **_volume(512)},
        # a large space in fine voxels: 2048^3 domain of 5 mm bf16 voxels in the block hash, faster camera
        {"name": "track_sparse_2048", "kind": "track", "width": 640, "height": 480, "frames": 12, "in_flight": 2,
         **_volume(2048, "bf16", sparse=True), "voxel_m": 0.005},
        # an interactive preview: small frames with colour, every result waited for before the next frame
        {"name": "track_color_256", "kind": "track", "width": 320, "height": 240, "frames": 8, "in_flight": 0,
         **_volume(256, "int16", color=True, rule="classic")},
        # several recordings reconstructed side by side on one GPU
        {"name": "batch_6", "kind": "batch", "width": 640, "height": 480, "frames": 6, "members": 6},
        # frames whose poses are known already, with colour, into 384^3 int16 voxels
        {"name": "fuse_color_384", "kind": "fuse", "width": 640, "height": 480, "frames": 10,
         **_volume(384, "int16", color=True)},
        # one view of a finished 512^3 model
        {"name": "render_512", "kind": "render", "width": 640, "height": 480, "mapped": 8, **_volume(512)},
        # a larger, odd-sized view of an odd-sized volume under the stricter corner rule
        {"name": "render_ragged", "kind": "render", "width": 1001, "height": 747, "mapped": 5,
         **_volume(333, "bf16", res_y=257, res_z=301), "all_corners": True, "cell_normals": True},
        # one frame's pyramid
        {"name": "pyramid_480", "kind": "pyramid", "width": 640, "height": 480},
        # the finest tracking level: ten Gauss-Newton steps
        {"name": "icp_480", "kind": "icp", "width": 640, "height": 480, "steps": 10},
        # the smallest call: one sweep of the coarsest level
        {"name": "sweep_120", "kind": "icp", "width": 160, "height": 120, "steps": 0},
        # the model of a finished scan as a mesh
        {"name": "mesh_512", "kind": "mesh", "width": 640, "height": 480, "mapped": 8, "min_weight": 2.0,
         **_volume(512)},
        # training the warm start at its usual batch
        {"name": "train_64", "kind": "train", "batch": 64, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_volume(rng, lo, hi):
    res = _log(rng, lo, hi)
    v = _volume(res, rng.choice(["float", "float", "int16", "bf16"]), rng.random() < 0.3,
                rng.choice(["angle", "angle", "classic"]), band=rng.random() < 0.2,
                res_y=max(8, int(res * rng.uniform(0.75, 1.0))), res_z=max(8, int(res * rng.uniform(0.75, 1.0))))
    v["all_corners"] = rng.random() < 0.25
    v["cell_normals"] = rng.random() < 0.25
    return v


def _draw_image(rng, lo, hi):
    width = _log(rng, lo, hi)
    return {"width": width, "height": max(48, int(width * rng.uniform(0.6, 0.8)))}


def draw(rng):
    kind = rng.choice(["track", "track", "track", "sparse", "batch", "fuse", "render", "render", "pyramid", "icp",
                       "icp", "mesh", "train"])
    if kind == "track":
        return {"kind": "track", **_draw_image(rng, 200, 800), "frames": rng.randint(4, 16),
                "in_flight": rng.choice([0, 2, 3]), **_draw_volume(rng, 128, 512)}
    if kind == "sparse":
        res = _log(rng, 512, 2048)
        return {"kind": "track", "width": 640, "height": 480, "frames": rng.randint(4, 12), "in_flight": 2,
                **_volume(res, rng.choice(["float", "int16", "bf16"]), sparse=True), "voxel_m": 10.24 / res}
    if kind == "batch":
        return {"kind": "batch", **_draw_image(rng, 320, 640), "frames": rng.randint(3, 6),
                "members": rng.randint(2, 6)}
    if kind == "fuse":
        return {"kind": "fuse", **_draw_image(rng, 200, 1000), "frames": rng.randint(3, 12),
                **_draw_volume(rng, 128, 512)}
    if kind == "render":
        return {"kind": "render", **_draw_image(rng, 100, 1280), "mapped": rng.randint(2, 8),
                **_draw_volume(rng, 128, 512)}
    if kind == "pyramid":
        return {"kind": "pyramid", **_draw_image(rng, 160, 1920)}
    if kind == "icp":
        return {"kind": "icp", **_draw_image(rng, 100, 1000), "steps": rng.choice([0, rng.randint(2, 12)])}
    if kind == "mesh":
        return {"kind": "mesh", "width": 640, "height": 480, "mapped": rng.randint(3, 8),
                "min_weight": rng.choice([0.0, 2.0]), **_draw_volume(rng, 128, 512)}
    return {"kind": "train", "batch": 8 * rng.randint(1, 8), "steps": rng.randint(2, 12)}


# ---- inputs ------------------------------------------------------------------------------
def _intrinsics(width, height):
    focal = synthetic.FX * width / 640.0
    return abi.Intrinsics(focal, focal, 0.5 * (width - 1), 0.5 * (height - 1))


def _frames(seed, count, width, height, step_m=0.01, step_deg=0.5, color=False):
    """(poses [count, 4, 4], uint16 depth and RGBA8 colour frames on the GPU) of a seeded sequence: the noise,
    dropout and clipping of kinectfusion_b200.synthetic at any image size."""
    rng = np.random.default_rng(seed)
    scene = synthetic.make_scene(rng)
    poses = synthetic.make_trajectory(rng, count, step_m, step_deg)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = _intrinsics(width, height)
    u, v = torch.meshgrid(torch.arange(width, dtype=torch.float64, device="cuda"),
                          torch.arange(height, dtype=torch.float64, device="cuda"), indexing="xy")
    rays = torch.stack([(u - k.cx) / k.fx, (v - k.cy) / k.fy, torch.ones_like(u)], dim=-1)
    spheres, boxes = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in (scene.spheres, scene.boxes))
    albedo = torch.tensor(scene.albedo.astype(np.int64), device="cuda")
    packed = (albedo[:, 0] | (albedo[:, 1] << 8) | (albedo[:, 2] << 16) | (-1 << 24)).to(torch.int32)
    depth, colors = [], []
    for pose in poses:
        z, pid = synthetic._render_torch(rays, spheres, boxes, torch.tensor(pose, device="cuda"))
        sigma = 0.0012 + 0.0019 * (z - 0.4) ** 2
        noisy = z + sigma * torch.randn(z.shape, generator=gen, dtype=torch.float64, device="cuda")
        edge = torch.zeros_like(z, dtype=torch.bool)
        for shift in ((0, 1), (0, -1), (1, 0), (-1, 0)):
            zn, pn = torch.roll(z, shift, (0, 1)), torch.roll(pid, shift, (0, 1))
            edge |= (pn != pid) & ((zn - z).abs() > 0.05)
        drop = torch.rand(z.shape, generator=gen, device="cuda") < 0.02
        valid = torch.isfinite(noisy) & (noisy >= 0.4) & (noisy <= 4.0) & ~edge & ~drop
        raw = torch.where(valid, torch.round(noisy * synthetic.DEPTH_SCALE), torch.zeros_like(noisy))
        depth.append(raw.to(torch.int32).to(torch.uint16))
        if color:
            colors.append(packed[pid.clamp(min=0)])
    return poses, torch.stack(depth), torch.stack(colors) if color else None


def _pipeline(case):
    res = (case["res"], case["res_y"], case["res_z"])
    vs = case["voxel_m"]
    config = kf.pipeline_config(
        res, vs, (-0.5 * res[0] * vs, -0.5 * res[1] * vs, -0.5), max(0.05, 3.0 * vs), voxel=VOXELS[case["voxel"]],
        color=abi.KF_COLOR_FLOAT if case["color"] else abi.KF_COLOR_NONE, rule=RULES[case["rule"]],
        storage=abi.KF_STORAGE_SPARSE if case["sparse"] else abi.KF_STORAGE_DENSE,
        integration_mode=abi.KF_INTEGRATION_BAND if case["band"] else abi.KF_INTEGRATION_FULL,
        raycast_corner_policy=abi.KF_CORNERS_REQUIRE_ALL if case["all_corners"] else abi.KF_CORNERS_SKIP_MISSING,
        raycast_cell_gradient_normals=1 if case["cell_normals"] else 0)
    return kf.Pipeline(config)


def _inverse(pose):
    inv = np.eye(4)
    inv[:3, :3] = pose[:3, :3].T
    inv[:3, 3] = -pose[:3, :3].T @ pose[:3, 3]
    return inv


def _build(pyramid, depth, k):
    """The pyramid of a depth frame in device memory."""
    h, w = depth.shape
    levels = C.c_uint32()
    abi.check(lib().kf_pyramid_build(pyramid.handle, C.c_void_p(depth.data_ptr()), w, h, k, abi.KF_MEMORY_DEVICE,
                                     C.byref(levels)))
    return levels.value


def _fuse(pipeline, pyramid, depth, color, k, pose):
    """Pyramid and integration of one frame in device memory at a known pose."""
    h, w = depth.shape
    _build(pyramid, depth, k)
    level = pyramid.level(0)
    view = abi.FrameView(C.c_void_p(depth.data_ptr()), None if color is None else C.c_void_p(color.data_ptr()),
                         level.normals, w, h, k, abi.rigid_from_matrix(_inverse(pose)), abi.KF_MEMORY_DEVICE)
    abi.check(lib().kf_pipeline_integrate(pipeline.handle, C.byref(view)))


def _render(pipeline, maps, k, pose):
    c2w = pose if isinstance(pose, abi.Rigid) else abi.rigid_from_matrix(pose)
    camera = abi.RaycastCamera(k, maps.width, maps.height, c2w)
    abi.check(lib().kf_pipeline_raycast(pipeline.handle, C.byref(camera), C.byref(maps.view())))
    return {"points": maps.points, "normals": maps.normals, "colors": maps.colors}


class _Device:
    """A device buffer of the library as __cuda_array_interface__ (no copy); a tensor made from it keeps `owner`,
    whose buffer it is, alive."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (ptr, False), "version": 3}


def _levels(pyramid, count):
    out = []
    for i in range(count):
        v = pyramid.level(i)
        shape = (v.height, v.width)
        out.append({"depth": torch.as_tensor(_Device(pyramid, v.depth, shape, "<i2"), device="cuda"),
                    "vertices": torch.as_tensor(_Device(pyramid, v.vertices, shape + (3,), "<f4"), device="cuda"),
                    "normals": torch.as_tensor(_Device(pyramid, v.normals, shape + (3,), "<f4"), device="cuda")})
    return out


def _pose(r):
    return [*r.r, *r.t]


def _member(case, i):
    """Sequence i of a batch: resolutions and voxel types in turn."""
    return _volume((128, 192, 256, 384, 512)[(3 * i + 1) % 5], ("int16", "bf16")[i % 2])


def _train_samples(seed, count):
    """Net inputs [count, 60, 80, 2] and targets [count, 6]: neighbouring views of a scene at 80x60, either
    played forwards or backwards, and the scaled twist between them."""
    poses, depth, _ = _frames(seed, count + 1, 80, 60, 0.004, 0.3)
    metres = depth.to(torch.float32) / synthetic.DEPTH_SCALE
    sign = np.random.default_rng(seed).integers(0, 2, count)
    inputs = torch.empty((count, 60, 80, 2), dtype=torch.float32, device="cuda")
    targets = np.empty((count, 6), dtype=np.float32)
    for i in range(count):
        a, b = (i, i + 1) if sign[i] else (i + 1, i)
        both = (metres[a] > 0) & (metres[b] > 0)
        mean = metres[a].sum() / (metres[a] > 0).sum().clamp(min=1)
        inputs[i, ..., 0] = torch.where(metres[b] > 0, metres[b] - mean, 0.0)
        inputs[i, ..., 1] = torch.where(both, (10.0 * (metres[b] - metres[a])).clamp(-1.0, 1.0), 0.0)
        targets[i] = 50.0 * learned.twist_between(poses[a], poses[b])
    return inputs.to(torch.bfloat16), torch.from_numpy(targets).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        learner = learned.Learner(batch_capacity=64, seed=seed & 0xFFFF)
        inputs, targets = _train_samples(seed, case["batch"])
        return {"case": case, "learner": learner, "inputs": inputs, "targets": targets,
                "losses": torch.zeros(case["steps"], device="cuda")}
    w, h = case["width"], case["height"]
    k = _intrinsics(w, h)
    s = {"case": case, "k": k}
    if kind == "batch":
        pipelines, s["frames"], s["maps"] = [], [], []
        for i in range(case["members"]):
            pipelines.append(_pipeline(_member(case, i)))
            s["frames"].append(_frames(seed + 1000 * i, case["frames"], w, h)[1])
            s["maps"].append(DeviceSurfaceMaps(w, h))
        s["batch"] = kf.Batch(pipelines, k)
        return s
    if kind == "track":
        _, depth, color = _frames(seed, case["frames"], w, h, *((0.02, 1.0) if case["sparse"] else (0.01, 0.5)),
                                  color=case["color"])
        s["depth"] = depth.cpu().numpy()
        s["color"] = None if color is None else color.cpu().numpy().view(np.uint32)
        loop = PipelinedReconstruction if case["in_flight"] else kf.Reconstruction
        s["loop"] = loop(_pipeline(case), k)
        s["maps"] = DeviceSurfaceMaps(w, h)
        return s
    pyramid = s["pyramid"] = kf.PyramidSource()
    if kind == "pyramid":
        s["depth"] = _frames(seed, 1, w, h)[1][0]
        return s
    if kind == "fuse":
        s["poses"], s["depth"], s["color"] = _frames(seed, case["frames"], w, h, color=case["color"])
        s["pipeline"], s["maps"] = _pipeline(case), DeviceSurfaceMaps(w, h)
        return s
    # a mapped volume: frames of 640x480 at their known poses
    mapped = case.get("mapped", 3)
    volume = case if kind != "icp" else _volume(256)
    k640 = _intrinsics(640, 480)
    poses, depth, color = _frames(seed, mapped + 1, 640, 480, color=volume["color"])
    pipeline = s["pipeline"] = _pipeline(volume)
    for i in range(mapped):
        _fuse(pipeline, pyramid, depth[i], None if color is None else color[i], k640, poses[i])
    s["maps"] = DeviceSurfaceMaps(w, h)
    s["pose"] = poses[mapped - 1]
    if kind == "icp":
        # the model at the last fused pose; the live frame one camera step later, and its start pose
        s["model"] = _render(pipeline, s["maps"], k, s["pose"])
        live = _frames(seed, mapped + 1, w, h)[1][mapped]
        _build(pyramid, live, k)
        s["live"] = pyramid.level(0)
        s["tracker"] = kf.ProjectiveIcpTracker()
    elif kind == "render":
        s["pose"] = poses[mapped]
    elif kind == "mesh":
        # the program's own mesh arrays, for up to 120 m^2 of surface
        most = int(120.0 / case["voxel_m"] ** 2)
        s["mesh"] = {"positions": np.zeros((most, 3), np.float32), "normals": np.zeros((most, 3), np.float32),
                     "colors": np.zeros((most, 3), np.float32), "triangles": np.zeros((2 * most, 3), np.uint32)}
    return s


# ---- one pass ----------------------------------------------------------------------------
def _run_track(s):
    case, loop = s["case"], s["loop"]
    # a new sequence: an empty volume, the start pose, no frames yet
    loop.pipeline.reset(wait=False)
    loop.frames, loop.pose = 0, abi.rigid_from_matrix(np.eye(4))
    loop.trajectory.clear()
    loop.results.clear()
    for i in range(case["frames"]):
        color = None if s["color"] is None else s["color"][i]
        if not case["in_flight"]:
            loop.process(s["depth"][i], color)
            continue
        loop.submit(s["depth"][i], color)
        if i + 1 >= case["in_flight"]:
            loop.next_result()
    while len(loop.results) < case["frames"]:
        loop.next_result()
    return {"poses": np.array([_pose(r.camera_to_world) for r in loop.results], dtype=np.float32),
            "status": np.array([[r.tracked, *r.status, *r.iterations, *r.correspondences] for r in loop.results],
                               dtype=np.int64),
            "view": _render(loop.pipeline, s["maps"], s["k"], loop.pose)}


def _run_batch(s):
    case, batch = s["case"], s["batch"]
    start = abi.rigid_from_matrix(np.eye(4))
    for p, t in zip(batch.pipelines, batch.trackers):
        p.reset(wait=False)
        abi.check(lib().kf_frame_set_pose(p.handle, t.handle, C.byref(start)))
    batch.frames = [0] * case["members"]
    for f in range(case["frames"]):
        batch.step([d[f].data_ptr() for d in s["frames"]], case["width"], case["height"])
    out = []
    for i, p in enumerate(batch.pipelines):
        r = batch.result(i)
        out.append({"pose": np.array(_pose(r.camera_to_world), dtype=np.float32),
                    "status": np.array([r.tracked, *r.status, *r.iterations, *r.correspondences], dtype=np.int64),
                    "view": _render(p, s["maps"][i], s["k"], r.camera_to_world)})
    return out


def _run_fuse(s):
    s["pipeline"].reset(wait=False)
    for i in range(s["case"]["frames"]):
        color = None if s["color"] is None else s["color"][i]
        _fuse(s["pipeline"], s["pyramid"], s["depth"][i], color, s["k"], s["poses"][i])
    return {"observed": s["pipeline"].observed_voxel_count(),
            "view": _render(s["pipeline"], s["maps"], s["k"], s["poses"][-1])}


def _run_icp(s):
    case, model, live = s["case"], s["model"], s["live"]
    points, normals = C.c_void_p(model["points"].data_ptr()), C.c_void_p(model["normals"].data_ptr())
    w, h = case["width"], case["height"]
    camera, to_model = abi.rigid_from_matrix(s["pose"]), abi.rigid_from_matrix(_inverse(s["pose"]))
    sums = np.empty(29, dtype=np.float32)
    if case["steps"] == 0:
        count = C.c_uint64()
        abi.check(lib().kf_icp_normal_equations(s["tracker"].handle, C.byref(live), points, normals, w, h, s["k"],
                                                C.byref(camera), C.byref(to_model),
                                                sums.ctypes.data_as(C.c_void_p), C.byref(count)))
        return {"sums": sums, "count": count.value}
    out = abi.IcpOutcome()
    abi.check(lib().kf_icp_level(s["tracker"].handle, C.byref(live), points, normals, w, h, s["k"],
                                 C.byref(to_model), C.byref(camera), case["steps"], C.byref(out),
                                 sums.ctypes.data_as(C.c_void_p)))
    return {"pose": np.array(_pose(out.pose), dtype=np.float32), "sums": sums,
            "count": [out.status, out.iterations, out.correspondences]}


def _run_mesh(s):
    mesh = abi.Mesh()
    abi.check(lib().kf_pipeline_extract_mesh(s["pipeline"].handle, s["case"]["min_weight"], C.byref(mesh)))
    counts = [mesh.vertex_count, mesh.triangle_count]
    for name, own in s["mesh"].items():
        n = counts[name == "triangles"]
        if n:
            own[:n] = np.ctypeslib.as_array(getattr(mesh, name), (n, 3))
    lib().kf_mesh_free(C.byref(mesh))
    return {"counts": counts, **s["mesh"]}


def _run_train(s):
    learner = s["learner"]
    for i in range(s["case"]["steps"]):
        learner.train_step(s["inputs"], s["targets"], 1e-3, s["losses"][i])
    return {"weights": learner.params(), "losses": s["losses"]}


def run(state):
    kind = state["case"]["kind"]
    if kind == "track":
        return _run_track(state)
    if kind == "batch":
        return _run_batch(state)
    if kind == "fuse":
        return _run_fuse(state)
    if kind == "render":
        return _render(state["pipeline"], state["maps"], state["k"], state["pose"])
    if kind == "pyramid":
        return _levels(state["pyramid"], _build(state["pyramid"], state["depth"], state["k"]))
    if kind == "icp":
        return _run_icp(state)
    if kind == "mesh":
        return _run_mesh(state)
    return _run_train(state)


# ---- what a pass cannot do without ---------------------------------------------------------
def _fused_voxels(volume, band):
    """Voxels of one frame's update: the view frustum up to a mean surface depth of 2.3 m, or its band."""
    solid = 480.0 / 640.0 * (640.0 / synthetic.FX) ** 2
    metres3 = solid * (2.3 ** 2 * 2.0 * max(0.05, 3.0 * volume["voxel_m"]) if band else 2.3 ** 3 / 3.0)
    count = metres3 / volume["voxel_m"] ** 3
    return min(count, float(volume["res"]) * volume["res_y"] * volume["res_z"])


def _sequence_work(volume, frames, pixels):
    """Depth (and colour) read, voxels read and written per frame; the volume emptied and one view written."""
    voxel = 8 if volume["voxel"] == "float" else 4
    cell = voxel + (16 if volume["color"] else 0)
    fused = _fused_voxels(volume, volume["band"])
    per_frame = pixels * (6 if volume["color"] else 2) + 2 * cell * fused
    empty = 0 if volume["sparse"] else cell * volume["res"] * volume["res_y"] * volume["res_z"]
    return frames * per_frame + empty + 28 * pixels, frames * (60 * fused + 400 * pixels) + 600 * pixels


def work(case):
    kind = case["kind"]
    if kind == "train":
        macs = case["batch"] * sum(r * c * n for r, c, n in
                                   ((32, 18, 1200), (32, 288, 300), (64, 288, 80), (64, 576, 20), (256, 1280, 1),
                                    (6, 256, 1)))
        return {"bytes": case["steps"] * (case["batch"] * 19200 + 28 * 395000.0), "flops": 6.0 * case["steps"] * macs}
    pixels = case["width"] * case["height"]
    if kind == "batch":
        parts = [_sequence_work(_member(case, i), case["frames"], pixels) for i in range(case["members"])]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind in ("track", "fuse"):
        b, f = _sequence_work(case, case["frames"], pixels)
        return {"bytes": b, "flops": f}
    if kind == "render":
        return {"bytes": 28.0 * pixels + 8.0 * 8 * pixels, "flops": 600.0 * pixels}
    if kind == "pyramid":
        return {"bytes": 2.0 * pixels + 26.0 * pixels * (1 + 1 / 4 + 1 / 16), "flops": 25 * 20.0 * pixels}
    if kind == "icp":
        return {"bytes": 48.0 * pixels, "flops": max(1, case["steps"]) * 120.0 * pixels}
    # mesh: the voxels of the observed surface band, and its vertices and triangles in host memory
    band = _fused_voxels(case, True) * (4 + 4 * (case["voxel"] == "float"))
    cells = _fused_voxels(case, True) / (2.0 * max(3.0, 0.05 / case["voxel_m"]))
    return {"bytes": band + cells * (36 + 24), "flops": 60 * cells}


# ---- 64-bit restatements ---------------------------------------------------------------------
def _exact_pyramid(case, seed):
    """BilateralFilter, BlockDownsample, VertexProjection and NormalEstimation in 64 bits."""
    o = kf.pipeline.default_depth_options()
    k = _intrinsics(case["width"], case["height"])
    raw = _frames(seed, 1, case["width"], case["height"])[1][0].to(torch.float64)

    def metres(r):
        d = r / o.depth_scale
        return torch.where((r > 0) & (d >= o.min_depth - 1e-7) & (d <= o.max_depth + 1e-7), d, math.nan)

    m, rad = metres(raw), o.bilateral_radius
    top, bottom = torch.zeros_like(m), torch.zeros_like(m)
    h, w = m.shape
    pad = torch.nn.functional.pad(torch.stack([raw, m]), (rad,) * 4, value=math.nan)
    for dy in range(2 * rad + 1):
        for dx in range(2 * rad + 1):
            r, s = pad[0, dy:dy + h, dx:dx + w], pad[1, dy:dy + h, dx:dx + w]
            g = torch.exp(-0.5 * ((dx - rad) ** 2 + (dy - rad) ** 2) / o.bilateral_spatial_sigma ** 2
                          - 0.5 * (s - m) ** 2 / o.bilateral_depth_sigma ** 2)
            g = torch.where(torch.isnan(g), 0.0, g)
            top += g * torch.where(g > 0, r, 0.0)
            bottom += g
    depth = torch.where(bottom > 0, torch.floor(top / bottom + 0.5), 0.0)
    out = []
    for level in range(o.levels):
        h, w = depth.shape
        f = 0.5 ** level
        u, v = torch.meshgrid(torch.arange(w, dtype=torch.float64, device="cuda"),
                              torch.arange(h, dtype=torch.float64, device="cuda"), indexing="xy")
        z = metres(depth)
        p = torch.stack([(u - k.cx * f) * z / (k.fx * f), (v - k.cy * f) * z / (k.fy * f), z], -1)
        n = torch.full_like(p, math.nan)
        left, right, up, down = p[1:-1, :-2], p[1:-1, 2:], p[:-2, 1:-1], p[2:, 1:-1]
        c = torch.linalg.cross(down - up, right - left)
        # a difference of exactly the threshold is decided by the 32-bit quotients
        z32 = (depth.to(torch.float32) / o.depth_scale)
        jump = torch.tensor(o.max_normal_depth_jump, dtype=torch.float32)
        far = ((z32[1:-1, 2:] - z32[1:-1, :-2]).abs() > jump) | ((z32[2:, 1:-1] - z32[:-2, 1:-1]).abs() > jump)
        length = c.norm(dim=-1, keepdim=True)
        bad = far[..., None] | torch.isnan(p[1:-1, 1:-1, 2:]) | ~(length > 0)
        n[1:-1, 1:-1] = torch.where(bad, math.nan, c / length)
        out.append({"depth": None, "vertices": p, "normals": n})
        quad = depth[:h // 2 * 2, :w // 2 * 2].reshape(h // 2, 2, w // 2, 2).permute(0, 2, 1, 3).reshape(h // 2, w // 2, 4)
        count = (quad > 0).sum(-1)
        hi, lo = quad.amax(-1), torch.where(quad > 0, quad, math.inf).amin(-1)
        hi32, lo32 = (x.to(torch.float32) / o.depth_scale for x in (hi, lo))
        keep = (count > 0) & ~((hi32 - lo32) > torch.tensor(o.max_downsample_depth_jump, dtype=torch.float32))
        mean = torch.floor((quad.sum(-1) + count // 2) / count.clamp(min=1))
        depth = torch.where(keep, mean, 0.0)
    return out


def _exact_icp(case, seed):
    """The normal equations, or the Gauss-Newton steps on them, in 64 bits over the same maps."""
    s = prepare(case, seed)
    live = _levels(s["pyramid"], 1)[0]
    lv, ln = (live[n].to(torch.float64).reshape(-1, 3) for n in ("vertices", "normals"))
    mp, mn = (s["model"][n].to(torch.float64).reshape(-1, 3) for n in ("points", "normals"))
    w, h, k = case["width"], case["height"], s["k"]
    o = kf.pipeline.default_icp_options()

    def rounded(m):
        """The pose as the call takes it: 32-bit values."""
        return torch.tensor(np.asarray(abi.matrix_from_rigid(abi.rigid_from_matrix(m)), dtype=np.float64), device="cuda")

    model = rounded(_inverse(s["pose"]))

    def sweep(cam):
        src = lv @ cam[:3, :3].T + cam[:3, 3]
        sim = src @ model[:3, :3].T + model[:3, 3]
        px = torch.floor(k.fx * sim[:, 0] / sim[:, 2] + k.cx + 0.5)
        py = torch.floor(k.fy * sim[:, 1] / sim[:, 2] + k.cy + 0.5)
        ok = torch.isfinite(sim).all(-1) & torch.isfinite(ln).all(-1) & (sim[:, 2] > 0)
        ok &= (px >= 0) & (py >= 0) & (px < w) & (py < h)
        at = torch.where(ok, py * w + px, 0.0).long()
        q, n = mp[at], mn[at]
        sn = ln @ cam[:3, :3].T
        sn = sn / sn.norm(dim=-1, keepdim=True)
        dist = (src - q).norm(dim=-1)
        ok &= torch.isfinite(q).all(-1) & torch.isfinite(n).all(-1)
        ok &= ~(dist > o.max_point_distance) & ~((sn * n).sum(-1) < o.min_normal_dot)
        src, q, n, dist = src[ok], q[ok], n[ok], dist[ok]
        j = torch.cat([torch.linalg.cross(src, n), n], -1)
        r = (n * (q - src)).sum(-1)
        return j.T @ j, j.T @ r, dist.sum(), (r * r).sum()

    def flat(a, b, d, e):
        iu = torch.triu_indices(6, 6, device="cuda")
        return torch.cat([a[iu[0], iu[1]], b, torch.stack([d, e])]).cpu().numpy()

    cam = rounded(s["pose"])
    if case["steps"] == 0:
        return {"sums": flat(*sweep(cam)), "count": None}
    sums = None
    for _ in range(case["steps"]):
        a, b, d, e = sweep(cam)
        sums = flat(a, b, d, e)
        x = torch.linalg.solve(a, b).cpu().numpy()
        turn = np.eye(4)
        turn[:3, :3], turn[:3, 3] = learned.so3_exp(x[:3]), x[3:]
        cam = torch.tensor(turn, device="cuda") @ cam
        if np.linalg.norm(x[3:]) < o.min_update_translation and np.linalg.norm(x[:3]) < o.min_update_rotation:
            break
    c = cam.cpu().numpy()
    return {"pose": np.concatenate([c[:3, :3].reshape(-1), c[:3, 3]]), "sums": sums, "count": None}


def _exact_train(case, seed):
    """The network, its loss, gradients and Adam steps in 64 bits with torch autograd."""
    s = prepare(case, seed)
    w = torch.tensor(s["learner"].params().astype(np.float64), device="cuda")
    convs = [(2, 32, 24), (32, 32, 288), (32, 64, 288), (64, 64, 576)]
    first, second = torch.zeros_like(w), torch.zeros_like(w)
    x = s["inputs"].to(torch.float64).permute(0, 3, 1, 2)
    target, losses = s["targets"].to(torch.float64), []
    for step in range(1, case["steps"] + 1):
        w.requires_grad_(True)
        at, hid = 0, x
        for cin, cout, cols in convs:
            weight = w[at:at + cout * cols].reshape(cout, cols)[:, :cin * 9].reshape(cout, cin, 3, 3)
            at += cout * cols
            hid = torch.relu(torch.nn.functional.conv2d(hid, weight, w[at:at + cout], stride=2, padding=1))
            at += cout
        hid = hid.permute(0, 2, 3, 1).reshape(case["batch"], 1280)
        hid = torch.relu(hid @ w[at:at + 256 * 1280].reshape(256, 1280).T + w[at + 327680:at + 327936])
        at += 327936
        out = hid @ w[at:at + 6 * 256].reshape(6, 256).T + w[at + 1536:at + 1542]
        loss = ((out - target) ** 2).sum() / case["batch"]
        g, = torch.autograd.grad(loss, w)
        losses.append(loss.detach())
        with torch.no_grad():
            first = 0.9 * first + 0.1 * g
            second = 0.999 * second + 0.001 * g * g
            w = w - 1e-3 * (first / (1 - 0.9 ** step)) / (torch.sqrt(second / (1 - 0.999 ** step)) + 1e-8)
    return {"weights": w.cpu().numpy(), "losses": torch.stack(losses)}


def exact(case, seed):
    restated = {"pyramid": _exact_pyramid, "icp": _exact_icp, "train": _exact_train}.get(case["kind"])
    return None if restated is None else restated(case, seed)
