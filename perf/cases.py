"""What the renderer is timed on: renders, ray queries and the guiding network, each through the
public Python entry points, over the range of sizes, scenes and options that programs use.

Scenes come from the repository's own seeded writers; a scene file is written once into the
temporary folder and loaded by every prepare(), as a program loads the scene it renders.
A case's seed moves the camera a little and picks the random streams (or the rays, weights and
records), so that another seed is another input.
"""
from __future__ import annotations

import json
import math
import os
import random
import tempfile

import numpy as np
import torch

import wurstrenderer_b200 as wr
from wurstrenderer_b200 import scenes


def listed():
    return [
        # an interactive preview after a camera move: one sample per pixel of a small frame of the
        # Cornell box; launches, host work and the length of the bounce chain are what it costs
        {"name": "box_preview", "kind": "render", "scene": "box", "width": 64, "height": 48, "spp": 1, "vertices": 10},
        # an ordinary small still: the 256x256 Cornell box
        {"name": "box_still", "kind": "render", "scene": "box", "width": 256, "height": 256, "spp": 16,
         "vertices": 10},
        # many uneven jobs (cameras, resolutions, sample counts) over one scene in one call
        {"name": "box_jobs", "kind": "jobs", "scene": "box", "jobs": 24, "job_seed": 1003, "most_spp": 64,
         "vertices": 14},
        # the benchmark's frame: 1,162,250 triangles, four area lights, 64 samples per pixel
        {"name": "terrain_1m", "kind": "render", "scene": "terrain", "grid": 512, "spheres": 2000, "width": 1024,
         "height": 512, "spp": 64, "vertices": 18},
        # an odd-sized draft frame into device memory on the tree that the device builds
        {"name": "terrain_draft", "kind": "render", "scene": "terrain", "grid": 256, "spheres": 600, "width": 637,
         "height": 359, "spp": 5, "vertices": 18, "lbvh": True, "device": True},
        # outdoors: equirectangular sky with suns beside 16 area lights, long paths, sharp Phong lobes
        {"name": "sky", "kind": "render", "scene": "sky", "grid": 384, "spheres": 2500, "width": 960, "height": 540,
         "spp": 12, "vertices": 26},
        # an indoor frame with the scene's trained network as its (frozen) proposal
        {"name": "room_guided", "kind": "render", "scene": "room", "width": 512, "height": 512, "spp": 8,
         "vertices": 10, "guided": True},
        # the light tracer: every connection splats
        {"name": "objects_splat", "kind": "render", "scene": "objects", "width": 320, "height": 240, "spp": 32,
         "vertices": 8, "integrator": "light_splatting"},
        # smooth low-poly objects as Phong tessellation patches (FP64 ray-patch tests)
        {"name": "patches", "kind": "render", "scene": "patches", "spheres": 700, "width": 640, "height": 320,
         "spp": 4, "vertices": 18},
        # ray queries from a program's own arrays: first hits with normals, then occlusion
        {"name": "rays_terrain", "kind": "rays", "scene": "terrain", "grid": 256, "spheres": 600, "rays": 1000003},
        # the guiding network on a program's own points
        {"name": "guide_points", "kind": "guide_eval", "scene": "box", "rows": 200003},
        # online training: Adam steps on one pass's records at the renderer's own minibatch size
        {"name": "guide_steps", "kind": "guide_train", "scene": "box", "records": 16384, "batch": 16384, "steps": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["box", "box", "terrain", "terrain", "sky", "room", "objects", "patches", "jobs", "rays",
                       "guide_eval", "guide_train"])
    if kind == "guide_eval":
        return {"kind": kind, "scene": "box", "rows": _log_int(rng, 100, 400000)}
    if kind == "guide_train":
        n = _log_int(rng, 500, 32768)
        return {"kind": kind, "scene": "box", "records": n, "batch": n if rng.random() < 0.5 else max(1, n // 3),
                "steps": rng.randint(1, 40)}
    if kind == "rays":
        if rng.random() < 0.5:
            return {"kind": kind, "scene": "box", "rays": _log_int(rng, 1000, 1500000)}
        return {"kind": kind, "scene": "terrain", "grid": 256, "spheres": 600, "rays": _log_int(rng, 1000, 1500000)}
    if kind == "jobs":
        return {"kind": kind, "scene": "box", "jobs": rng.randint(2, 20), "job_seed": rng.randint(1, 10**6),
                "most_spp": _log_int(rng, 4, 40), "vertices": rng.randint(4, 14)}
    # a frame: its shape, then samples up to a bounded number of paths
    width = _log_int(rng, 32, 1280)
    height = max(16, int(width * rng.uniform(0.5, 1.0)))
    most = {"box": 6e6, "terrain": 8e6, "sky": 6e6, "room": 1.5e6, "objects": 6e6, "patches": 6e5}[kind]
    case = {"kind": "render", "scene": kind, "width": width, "height": height,
            "spp": _log_int(rng, 1, max(1.0, min(256.0, most / (width * height)))), "vertices": rng.randint(3, 20)}
    if kind in ("terrain", "sky"):
        case.update(grid=256, spheres=600)
    if kind == "terrain" and rng.random() < 0.4:
        case["lbvh"] = True
    if kind == "patches":
        case["spheres"] = 700
    if kind == "room" and rng.random() < 0.6:
        case["guided"] = True
    if kind == "objects":
        case["integrator"] = rng.choice(["light_splatting", "primitive_path_tracer", "nextevent_path_tracer"])
    elif rng.random() < 0.3:
        case["device"] = True
    return case


# ------------------------------------------------------------------ scenes ----
def _scene_file(case):
    """The case's scene file, written on its first use."""
    s = case["scene"]
    name = "_".join([s] + [str(case[k]) for k in ("grid", "spheres") if k in case])
    folder = os.path.join(tempfile.gettempdir(), "wurst_b200_scenes_%d" % os.getuid(), name)
    path = os.path.join(folder, name + ".json")
    if os.path.exists(path):
        return path
    os.makedirs(os.path.dirname(folder), exist_ok=True)
    new = tempfile.mkdtemp(dir=os.path.dirname(folder))
    if s == "box":
        scenes.write_cornell(new, name)
    elif s == "terrain":
        scenes.write_heightfield_spheres(new, name, n_grid=case["grid"], n_spheres=case["spheres"])
    elif s == "sky":
        scenes.write_full_combination(new, name, n_grid=case["grid"], n_spheres=case["spheres"])
    elif s == "room":
        scenes.write_spec(new, name, scenes.door_room_spec(), scenes.DOOR_ROOM_CAMERA, (1024, 1024), 64, 10)
    elif s == "objects":
        scenes.write_env_scene(new, name, env_size=(512, 256))
    elif s == "patches":
        scenes.write_heightfield_phong(new, name, n_spheres=case["spheres"])
    else:
        raise ValueError(s)
    try:
        os.rename(new, folder)
    except OSError:   # another process wrote it meanwhile
        pass
    return path


_CAMERAS = {"box": scenes.CORNELL_CAMERA, "terrain": scenes.HEIGHTFIELD_CAMERA, "sky": scenes.FULL_COMBINATION_CAMERA,
            "room": scenes.DOOR_ROOM_CAMERA, "objects": scenes.ENV_CAMERA, "patches": scenes.HEIGHTFIELD_CAMERA}

# (triangles, rays a path at least takes per vertex beyond the first two, bounding box of useful ray origins)
_FACTS = {"box": (36, 2.0, (-0.95, 0.05, -0.95, 0.95, 1.9, 0.95)), "room": (197782, 2.0, None),
          "objects": (1386, 0.4, None), "terrain": (1162250, 0.2, (-7.5, 0.4, -7.5, 7.5, 3.0, 7.5)),
          "sky": (495154, 0.1, None), "patches": (578250, 0.2, None)}


def _triangles(case):
    n = _FACTS[case["scene"]][0]
    if case["scene"] == "terrain":
        n = 2 * (case["grid"] - 1) ** 2 + 320 * case["spheres"] + 8
    elif case["scene"] == "sky":
        n = 2 * (case["grid"] - 1) ** 2 + 80 * case["spheres"] + 32
    elif case["scene"] == "patches":
        n = 2 * 511 ** 2 + 80 * case["spheres"] + 8
    return n


def _load(case):
    return wr.Scene.from_file(_scene_file(case), bvh_builder=wr.BVH_DEVICE_LBVH if case.get("lbvh") else wr.BVH_HOST_SAH)


def _moved_camera(case, rng):
    cam = dict(_CAMERAS[case["scene"]])
    cam["pos"] = [float(x + rng.uniform(-0.03, 0.03)) for x in cam["pos"]]
    cam["resolution"] = [case["width"], case["height"]]
    return cam


def _jobs(case, rng, seed):
    jobs = scenes.batch_jobs(seed=case["job_seed"], n_jobs=case["jobs"], num_path_vertices=case["vertices"])
    for k, j in enumerate(jobs):
        w = j["camera"]["resolution"][0]
        j["camera"]["resolution"] = [w, max(8, w * 3 // 4 - k % 3)]
        j["camera"]["fovy"] = float(rng.uniform(50.0, 70.0))
        j["num_spp"] = max(1, min(j["num_spp"], case["most_spp"]))
        j["seed"] = (seed * 7919 + k) & 0x7fffffff
    return jobs


def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _rays(case, rng):
    """Half camera rays, half rays between random points of the scene; (n, 8) as the queries take them."""
    n = case["rays"]
    cam = _CAMERAS[case["scene"]]
    pos, look = np.array(cam["pos"]), np.array(cam["lookat"])
    z = look - pos
    z /= np.linalg.norm(z)
    x = np.cross(np.array(cam["up"]), z)
    x /= np.linalg.norm(x)
    y = np.cross(z, x)
    half = n // 2
    f = math.tan(math.radians(cam["fovy"]) / 2)
    uv = rng.uniform(-f, f, (half, 2))
    rays = np.zeros((n, 8), np.float32)
    box = _FACTS[case["scene"]][2]
    d = z + uv[:, :1] * x + uv[:, 1:] * y
    rays[:half, 0:3] = pos
    rays[:half, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[half:, 0:3] = rng.uniform(box[:3], box[3:], (n - half, 3))
    rays[half:, 4:7] = _unit(rng, n - half)
    rays[:, 3] = 1e-4
    rays[:, 7] = np.inf
    return rays


def _net(rng):
    w = (rng.normal(size=(5, 64, 64)) / 8.0).astype(np.float32)
    w[:4, 63, :] = 0.0      # the constant unit of every hidden layer
    w[:4, 63, 63] = 1.0
    return w


def _guide_box_points(rng, box, n):
    lo, inv = box    # as Scene.guide_box gives them
    return (np.float64(lo) + rng.uniform(0.02, 0.98, (n, 3)) / np.float64(inv)).astype(np.float32)


def _records(rng, box, n):
    """Training records as the tracer leaves them: point, weight, normal, outgoing and sampled direction."""
    rec = np.zeros((n, 5, 4), np.float32)
    rec[:, 0, :3] = _guide_box_points(rng, box, n)
    rec[:, 0, 3] = rng.exponential(1.0, n) * (rng.uniform(size=n) >= 0.2)
    rec[:, 1, :3] = _unit(rng, n)
    rec[:, 2, :3] = _unit(rng, n)
    toward = np.array([0.0, 1.9, 0.0]) - rec[:, 0, :3] + 0.4 * rng.normal(size=(n, 3))
    rec[:, 3, :3] = toward / np.linalg.norm(toward, axis=1, keepdims=True)
    rec[:, 4, :3] = 1.0
    return rec.reshape(n, 20)


# ----------------------------------------------------------------- the cases ----
def prepare(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    scene = _load(case)
    state = {"case": case, "scene": scene, "kind": kind, "seed": int(rng.integers(1, 1 << 31))}
    if kind == "render":
        scene.set_camera(json.dumps(_moved_camera(case, rng)))
        if case.get("guided"):
            scene.guide_set_params(_net(rng))
        if case.get("device"):
            state["image"] = torch.empty(case["height"], case["width"], 3, dtype=torch.float64, device="cuda")
    elif kind == "jobs":
        state["jobs"] = _jobs(case, rng, seed)
    elif kind == "rays":
        state["rays"], state["shadow"] = _rays(case, rng), _rays(case, rng)
        state["shadow"][:, 7] = rng.uniform(0.1, 3.0, case["rays"])
    elif kind == "guide_eval":
        scene.guide_set_params(_net(rng))
        n = case["rows"]
        state["rows"] = np.concatenate([_guide_box_points(rng, scene.guide_box(), n), _unit(rng, n), _unit(rng, n)],
                                       1).astype(np.float32)
    elif kind == "guide_train":
        state["net"] = _net(rng)
        state["records"] = _records(rng, scene.guide_box(), case["records"])
    return state


def run(state):
    case, scene, kind = state["case"], state["scene"], state["kind"]
    if kind == "render":
        guiding = "frozen" if case.get("guided") else 0
        if case.get("device"):
            scene.render_device(state["image"].data_ptr(), spp=case["spp"], num_path_vertices=case["vertices"],
                                seed=state["seed"], guiding=guiding)
            return state["image"]
        return scene.render(spp=case["spp"], num_path_vertices=case["vertices"], seed=state["seed"],
                            integrator=case.get("integrator"), guiding=guiding)
    if kind == "jobs":
        return scene.render_batch(state["jobs"])
    if kind == "rays":
        geom, prim, t, normal = scene.trace_hits(state["rays"])
        _, _, _, uv = scene.trace_closest(state["rays"])
        return {"geom": geom, "prim": prim, "t": t, "normal": normal, "uv": uv,
                "occluded": scene.trace_occluded(state["shadow"])}
    if kind == "guide_eval":
        axis, sharpness, weight = scene.guide_eval(state["rows"])
        return {"axis": axis, "sharpness": sharpness, "weight": weight}
    scene.guide_reset(1)                       # a new network: optimiser state cleared
    scene.guide_set_params(state["net"])
    losses = scene.guide_train(state["records"], case["steps"], batch=case["batch"], lr=1e-3)
    return {"weights": scene.guide_params(), "losses": losses}


def work(case):
    kind = case["kind"]
    if kind == "guide_eval":    # 9 floats in, 40 out; five 64 x 64 layers
        return {"bytes": case["rows"] * 4 * 49 + 40960, "flops": case["rows"] * 37888.0}
    if kind == "guide_train":   # forward, input gradient and weight gradient
        rows = min(case["batch"], case["records"]) * case["steps"]
        return {"bytes": case["records"] * 80 + 2 * 81920, "flops": rows * 3 * 40960.0}
    ntri = _triangles(case)
    per_ray = 30.0 * math.log2(ntri) + 60.0      # one descent of box pairs and one triangle test
    scene_bytes = ntri * 36.0
    if kind == "rays":
        return {"bytes": scene_bytes + case["rays"] * (2 * 32 + 32 + 4 + 28.0), "flops": case["rays"] * 3 * per_ray}
    if kind == "jobs":
        shapes = _jobs(case, np.random.default_rng(0), 0)
        pixels = sum(j["camera"]["resolution"][0] * j["camera"]["resolution"][1] for j in shapes)
        paths = sum(j["camera"]["resolution"][0] * j["camera"]["resolution"][1] * j["num_spp"] for j in shapes)
    else:
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp"]
    rays = paths * (2.0 + _FACTS[case["scene"]][1] * max(0, case["vertices"] - 2))
    return {"bytes": scene_bytes + 24.0 * pixels, "flops": rays * per_ray}


# ------------------------------------------------------- in 64 bits, where there is one ----
def _encode(p01, n, wo):
    parts = [p01]
    for f in range(6):
        a = (2.0 ** f) * math.pi * p01
        parts += [torch.sin(a), torch.cos(a)]
    parts += [n, wo, torch.sin(math.pi * n), torch.cos(math.pi * n), torch.sin(math.pi * wo), torch.cos(math.pi * wo)]
    x = torch.cat(parts, 1)
    pad = torch.zeros(x.shape[0], 7, dtype=x.dtype)
    pad[:, 6] = 1.0
    return torch.cat([x, pad], 1)


def _lobes(layers, x):
    for l in range(5):
        x = x @ layers[l].T
        if l < 4:
            x = torch.relu(x)
    o = x[:, :40].reshape(-1, 8, 5)
    mu = o[..., :3] / o[..., :3].norm(dim=-1, keepdim=True)
    lam = torch.clamp(torch.nn.functional.softplus(o[..., 3]) + 0.5, max=5000.0)
    return mu, lam, torch.softmax(o[..., 4], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("guide_eval", "guide_train"):
        return None   # Monte Carlo images of the renderer's own random streams; first hits by number
    rng = np.random.default_rng([seed, 20])
    rng.integers(1, 1 << 31)
    net = torch.from_numpy(_net(rng)).double()
    lo, hi = _box_bounds()
    ext = hi - lo
    lo, inv = lo - 0.01 * ext, 1.0 / (1.02 * ext)
    if kind == "guide_eval":
        n = case["rows"]
        rows = torch.from_numpy(np.concatenate([_guide_box_points(rng, (lo.astype(np.float32), inv.astype(np.float32)), n),
                                                _unit(rng, n), _unit(rng, n)], 1).astype(np.float32)).double()
        out = []
        for at in range(0, n, 65536):
            r = rows[at:at + 65536]
            out.append(_lobes(net, _encode((r[:, :3] - torch.from_numpy(lo)) * torch.from_numpy(inv), r[:, 3:6], r[:, 6:9])))
        mu, lam, w = (torch.cat(x) for x in zip(*out))
        return {"axis": mu, "sharpness": lam, "weight": w}
    if case["batch"] != case["records"] or case["records"] * case["steps"] > 700000:
        return None   # minibatches in the library's own order; more than some seconds
    rec = torch.from_numpy(_records(rng, (lo.astype(np.float32), inv.astype(np.float32)), case["records"])).double()
    rec = rec.reshape(-1, 5, 4)
    c, d = torch.clamp(rec[:, 0, 3], max=100.0), rec[:, 3, :3]
    x = _encode((rec[:, 0, :3] - torch.from_numpy(lo)) * torch.from_numpy(inv), rec[:, 1, :3], rec[:, 2, :3])
    w = net.clone()
    m, v, losses = torch.zeros_like(w), torch.zeros_like(w), []
    for k in range(1, case["steps"] + 1):
        w.requires_grad_(True)
        mu, lam, weight = _lobes(w, x)
        cosine = (mu * d[:, None, :]).sum(-1)
        f = weight * lam / (2 * math.pi * -torch.expm1(-2 * lam)) * torch.exp(lam * (cosine - 1))
        loss = -(c * torch.log(f.sum(-1))).sum() / case["records"]
        g, = torch.autograd.grad(loss, w)
        losses.append(float(loss.detach()))
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            w = w - 1e-3 * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
            w[:4, 63, :] = 0.0
            w[:4, 63, 63] = 1.0
        w = w.detach()
    return {"weights": w, "losses": np.array(losses)}


def _box_bounds():
    """Bounds of the Cornell box's vertices, which the guiding features are scaled by."""
    points = np.concatenate([m.positions for m in scenes.cornell_spec().meshes]).astype(np.float64)
    return points.min(0), points.max(0)
