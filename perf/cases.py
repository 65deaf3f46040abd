"""The renderer's work as its users call it, from a 256 x 256 preview frame to a 1080p still.

Every case goes through the public Python classes (RendererKernel, BatchRenderer and the torch
function over DiffRenderer). Scenes are the repository's synthetic workloads; the seed moves the
camera, the sun and the random streams (and, for the sphere scenes, places and colours the spheres),
and geometry is compiled once per detail level, as a program that renders a scene more than once does.
Where a case carries launch tuning, the values are those the repository's tuners pick for that scene.
"""
import copy
import functools
import math
import sys

import numpy as np
import torch

if "dayflower-path-tracer_gb300" not in sys.path:
    sys.path.insert(0, "dayflower-path-tracer_gb300")

from dfpt import diff, synthetic  # noqa: E402
from dfpt.batch import BatchRenderer  # noqa: E402
from dfpt.kernel import RendererKernel  # noqa: E402
from dfpt.scene import SkyState, camera_set_resolution  # noqa: E402

# dfpt_set_tuning keys that a case may carry.
TUNING = ("primitive_culling", "trace_config", "tail_bounce", "tail_blocks", "pass_shadow_sort", "wide_samples", "shadow_defer")
RENDERERS = {"ambient_occlusion": 1, "path_tracer": 2, "ray_caster": 3, "ray_tracer": 5, "surface_normals": 6}


def listed():
    return [
        # The smallest preview: one frame of a few spheres; launches and latency count.
        dict(name="frame_spheres_256", kind="frames", scene="spheres", detail=0, width=256, height=256, frames=1),
        # The interactive loop on the headline scene, with the launch structure dfpt_tune_frame picks.
        dict(name="frames_mesh_1080p", kind="frames", scene="mesh", detail=100, width=1920, height=1080, frames=8,
             trace_config=17, tail_bounce=1, tail_blocks=4),
        # The same loop without tuning, in a window of odd size, on many instances and small lights.
        dict(name="frames_instances_odd", kind="frames", scene="instances", detail=20, width=1279, height=717, frames=8,
             primitive_culling=2),
        # A still of the headline scene: the wave settings the tuner picks, in a smaller wave (memory).
        dict(name="still_mesh_1080p", kind="still", scene="mesh", detail=100, width=1920, height=1080, passes=32,
             trace_config=17, wide_samples=16, shadow_defer=1),
        # A still with the defaults, odd in every size: 19 passes are two waves of 8 and one of 3.
        dict(name="still_mesh_odd", kind="still", scene="mesh", detail=37, width=641, height=479, passes=19),
        # No meshes: the primitive loop and the shading.
        dict(name="still_spheres_512", kind="still", scene="spheres", detail=0, width=512, height=512, passes=64, wide_samples=64),
        # Many primitives under the culling BVH.
        dict(name="still_instances_720p", kind="still", scene="instances", detail=30, width=1280, height=720, passes=24,
             primitive_culling=2, wide_samples=12, shadow_defer=1),
        # The editor's ray-cast view: the image and the buffer that a click picks a primitive from.
        dict(name="raycast_mesh_1080p", kind="view", renderer="ray_caster", scene="mesh", detail=100, width=1920, height=1080),
        # The other views of the same editor.
        dict(name="occlusion_mesh_odd", kind="view", renderer="ambient_occlusion", scene="mesh", detail=60, width=1003, height=601),
        dict(name="normals_object_640", kind="view", renderer="surface_normals", scene="object", detail=16, width=640, height=480),
        # A queue of small and middling scenes rendered together.
        dict(name="batch_of_12", kind="batch", scenes=12, triangles_max=60000, spp=16, resolution_max=512, capacity=1 << 22),
        # One step of inverse rendering: the image, a loss, and the gradient of every parameter.
        dict(name="inverse_512", kind="inverse", spheres=256, width=512, height=512, spp=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames", "frames", "still", "still", "still", "view", "batch", "inverse"])
    width = _log(rng, 160, 1920)
    height = max(96, int(width * rng.uniform(0.5, 0.8)))
    if rng.random() < 0.5:
        width, height = width // 8 * 8, height // 4 * 4
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 12), triangles_max=_log(rng, 2000, 60000), spp=rng.randint(4, 24),
                    resolution_max=rng.randint(128, 512), capacity=1 << rng.randint(20, 22))
    if kind == "inverse":
        return dict(kind=kind, spheres=rng.randint(9, 256), width=min(width, 512), height=min(height, 400), spp=rng.randint(2, 16))
    if kind == "view":
        renderer = rng.choice(["ray_caster", "ambient_occlusion", "surface_normals", "ray_tracer"])
        if rng.random() < 0.5:
            return dict(kind=kind, renderer=renderer, scene="object", detail=rng.randint(6, 24), width=min(width, 800), height=min(height, 600))
        return dict(kind=kind, renderer=renderer, scene="mesh", detail=_log(rng, 12, 60), width=width, height=height)
    scene = rng.choice(["mesh", "mesh", "mesh", "instances", "spheres"])
    detail = {"mesh": _log(rng, 12, 100), "instances": rng.randint(6, 20), "spheres": 0}[scene]
    case = dict(kind=kind, scene=scene, detail=detail, width=width, height=height)
    if scene == "instances":
        case["primitive_culling"] = rng.choice([1, 2, 2])
    if kind == "frames":
        case["frames"] = rng.randint(1, 8)
        if rng.random() < 0.6:
            case |= dict(trace_config=rng.choice([16, 17]), tail_bounce=rng.randint(0, 2), tail_blocks=rng.randint(2, 4),
                         pass_shadow_sort=rng.randint(0, 1))
    else:
        case["passes"] = rng.randint(2, 26)
        if rng.random() < 0.6:
            case |= dict(trace_config=rng.choice([16, 17]), wide_samples=rng.choice([4, 12, 16]), shadow_defer=rng.randint(0, 1))
    return case


# -- scenes ---------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=24)
def _compiled(scene, detail):
    if scene == "mesh":  # 722,242 triangles at detail 100
        return synthetic.mesh_scene(frequency=detail, grid=max(8, int(5.12 * detail)))[0::2]
    if scene == "instances":  # 40 meshes of 20 detail^2 triangles, 500 emitting triangles
        return synthetic.instances_scene(frequency=detail)[0::2]
    compiled, _, params = synthetic.batch_scene(detail, 20 * detail * detail, 640, 480)  # "object": a mesh on a plane
    return compiled, params


def _scene(case, seed):
    """(CompiledScene, SkyState, parameters) with the seed's camera, sun and random stream."""
    rng = np.random.default_rng(seed)
    if case["scene"] == "spheres":
        compiled, _, params, _ = synthetic.sphere_scene(seed, case["width"], case["height"])
    else:
        shared, params = _compiled(case["scene"], case["detail"])
        compiled = copy.copy(shared)
        compiled.camera = shared.camera.copy()
        compiled.camera[1:4] += rng.uniform(-0.3, 0.3, 3).astype(np.float32)
    camera_set_resolution(compiled.camera, case["width"], case["height"])
    azimuth, elevation = rng.uniform(0, 2 * np.pi), rng.uniform(0.5, 1.1)
    sun = (np.cos(elevation) * np.cos(azimuth), np.sin(elevation), np.cos(elevation) * np.sin(azimuth))
    sky = SkyState(tuple(float(v) for v in sun), float(rng.uniform(2.0, 4.0)))
    return compiled, sky, dict(params, seed=int(rng.integers(1, 1 << 31)))


def _batch_scenes(case, seed):
    """Triangle counts log-uniform from 1,000, square images, samples per pixel as given, half or double."""
    sizes = np.random.default_rng(case["scenes"])  # the mix belongs to the case, the streams to the seed
    rng = np.random.default_rng(seed)
    for _ in range(case["scenes"]):
        triangles = int(np.exp(sizes.uniform(np.log(1000), np.log(case["triangles_max"]))))
        side = int(sizes.integers(case["resolution_max"] // 4, case["resolution_max"] + 1))
        spp = max(1, int(case["spp"] * 2.0 ** sizes.integers(-1, 2)))
        yield triangles, side, spp, int(rng.integers(1, 1 << 31))


def prepare(case, seed):
    if case["kind"] == "batch":
        batch = BatchRenderer()
        for triangles, side, spp, stream in _batch_scenes(case, seed):
            compiled, params = _compiled("object", max(1, int(round(math.sqrt(triangles / 20)))))
            compiled = copy.copy(compiled)
            compiled.camera = camera_set_resolution(compiled.camera.copy(), side, side)
            rng = np.random.default_rng(stream)
            batch.add(compiled, side, side, spp, SkyState((0.5, float(rng.uniform(0.4, 1.0)), 0.5), 2.5), dict(params, seed=stream))
        batch.set_tuning("wave_capacity", case["capacity"])
        return dict(case=case, batch=batch)
    if case["kind"] == "inverse":
        compiled, params, _, truth, start = synthetic.inverse_scene(seed, case["width"], case["height"], case["spheres"])
        kernel = RendererKernel(compiled, SkyState(truth["sun_direction"], truth["turbidity"]), dict(params, seed=seed & 0xFFFFFF))
        kernel.update(case["width"], case["height"])
        kernel.set_tuning("wide_samples", case["spp"])
        rng = np.random.default_rng(seed)
        albedo = torch.tensor(start["albedo"] * rng.uniform(0.8, 1.2, start["albedo"].shape).astype(np.float32), requires_grad=True)
        parameters = [albedo, torch.zeros_like(albedo).requires_grad_(), torch.tensor(start["phong_exponent"], requires_grad=True),
                      torch.tensor(2.0, requires_grad=True), torch.tensor(start["sun_direction"], requires_grad=True)]
        target = torch.tensor(rng.uniform(0.0, 0.6, (case["height"], case["width"], 3)), dtype=torch.float32)
        return dict(case=case, kernel=kernel, renderer=diff.DiffRenderer(kernel), function=diff.render_function(),
                    parameters=parameters, target=target)
    compiled, sky, params = _scene(case, seed)
    kernel = RendererKernel(compiled, sky, dict(params, renderer_type=RENDERERS[case.get("renderer", "path_tracer")]))
    kernel.update(case["width"], case["height"])
    for key in TUNING:
        if key in case:
            kernel.set_tuning(key, case[key])
    return dict(case=case, kernel=kernel)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch = state["batch"]
        batch.render()
        return [batch.film(i) for i in range(len(batch.sizes))]
    if case["kind"] == "inverse":
        for p in state["parameters"]:
            p.grad = None
        image = state["function"].apply(state["renderer"], case["spp"], *state["parameters"])
        ((image - state["target"]) ** 2).sum().backward()
        return [image.detach()] + [p.grad for p in state["parameters"]]
    kernel = state["kernel"]
    kernel.clear()
    if case["kind"] == "frames":
        for _ in range(case["frames"]):
            kernel.execute(1)
        return kernel.film()
    if case["kind"] == "still":
        kernel.execute(case["passes"])
        return kernel.film()
    kernel.execute(1)
    # Per-pixel views take no random sums: the image's bytes are reproducible.
    if case["renderer"] == "surface_normals":
        return {"film": kernel.film()[0], "picked": kernel.primitive_offsets()}
    return {"image": kernel.get(), "picked": kernel.primitive_offsets()}


# -- the least a pass has to move and compute -----------------------------------------------------

def work(case):
    """Bytes: the scene once, the film or image once. Flops: for each ray, one root-to-leaf path of a
    balanced binary tree over the triangles (two boxes a level, 18 operations each), two triangle
    tests (45 each) and, for camera and bounce rays, 400 for surface, sampling and random numbers.
    Rays per sample as the renderer's counters report them for these scenes."""
    if case["kind"] == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for triangles, side, spp, _ in _batch_scenes(case, 0):
            total["bytes"] += triangles * 112.0 + side * side * 16.0
            total["flops"] += side * side * spp * (1.9 * (36 * math.log2(triangles) + 490) + 0.8 * (36 * math.log2(triangles) + 90))
        return total
    pixels = case["width"] * case["height"]
    if case["kind"] == "inverse":
        samples, primitives = pixels * case["spp"], case["spheres"] + 1
        closest, any_hit = 2.2, 1.2
        # Forward and replay of the same rays, without the replay's shadow rays.
        flops = samples * (2 * closest * (36 * math.log2(primitives) + 460) + any_hit * (36 * math.log2(primitives) + 60))
        return dict(bytes=pixels * 12.0 * 2 + primitives * 220.0, flops=flops)
    d = case["detail"]
    triangles = {"mesh": 20 * d * d + 2 * (max(8, int(5.12 * d)) - 1) ** 2, "instances": 800 * d * d + 500, "spheres": 4, "object": 20 * d * d}[case["scene"]]
    ray = 36 * math.log2(max(2, triangles)) + 90
    if case["kind"] == "view":
        rays = {"surface_normals": 1.0, "ray_caster": 1.8, "ambient_occlusion": 1.8, "ray_tracer": 1.8}[case["renderer"]]
        return dict(bytes=triangles * 112.0 + pixels * 8.0, flops=pixels * (rays * ray + 200))
    samples = pixels * (case["frames"] if case["kind"] == "frames" else case["passes"])
    closest, any_hit = {"mesh": (1.8, 0.8), "instances": (1.05, 0.05), "spheres": (2.0, 0.9)}[case["scene"]]
    return dict(bytes=triangles * 112.0 + pixels * 16.0, flops=samples * (closest * (ray + 400) + any_hit * ray))


# -- 64-bit values --------------------------------------------------------------------------------

def exact(case, seed):
    """The surface-normal view of a meshed object on a plane: every triangle against every camera ray.
    The path-traced films have no such value: each sample is a random path whose turns hang on 32-bit
    comparisons, and a 64-bit path soon takes other ones. The other views give bytes."""
    if case["kind"] != "view" or case["renderer"] != "surface_normals" or case["scene"] != "object":
        return None
    scene, sky, _ = _scene(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t64(a):
        return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)

    if not all(np.array_equal(m, np.eye(4)) for m in scene.primitives_world_to_object.reshape(-1, 4, 4).astype(np.float64)):
        return None
    w, h = case["width"], case["height"]
    cam = scene.camera.astype(np.float64)
    eye, U, V, W = (t64(cam[i:i + 3]) for i in (1, 7, 10, 13))
    x = (torch.arange(w, dtype=torch.float64, device=dev) + 0.5) / (cam[16] - 1) * 2 - 1
    y = (torch.arange(h, dtype=torch.float64, device=dev) + 0.5) / (cam[17] - 1) * 2 - 1
    gy, gx = torch.meshgrid(y, x, indexing="ij")
    d = W + U * (math.tan(math.radians(cam[4]) / 2) * gx.reshape(-1, 1)) + V * (math.tan(-math.radians(cam[5]) / 2) * gy.reshape(-1, 1))
    d = d / d.norm(dim=1, keepdim=True)
    n = len(d)
    best = torch.full((n,), 100000.0, dtype=torch.float64, device=dev)
    normal = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    hit = torch.zeros(n, dtype=torch.bool, device=dev)
    # Planes.
    p = scene.point3fs.astype(np.float64)
    v = scene.vector3fs.astype(np.float64)
    for kind, offset, _ in scene.primitives.reshape(-1, 3):
        if kind == 1:
            a = t64(p[scene.planes[offset]:scene.planes[offset] + 3])
            nn = t64(v[scene.planes[offset + 3]:scene.planes[offset + 3] + 3])
            t = ((a - eye) @ nn) / (d @ nn)
            ok = (t > 0.001) & (t < best)
            best, hit = torch.where(ok, t, best), hit | ok
            normal = torch.where(ok[:, None], nn.expand(n, 3), normal)
    # Triangles (Moller-Trumbore), a block of rays at a time.
    T = scene.triangles.reshape(-1, 12)
    corner = [t64(np.stack([p[T[:, k] + c] for c in range(3)], 1)) for k in range(3)]
    at = [t64(np.stack([v[T[:, 3 + k] + c] for c in range(3)], 1)) for k in range(3)]
    a, e0, e1 = corner[0], corner[1] - corner[0], corner[2] - corner[0]
    s = eye - a
    q = torch.linalg.cross(s, e0)
    te1q, e1xe0, sxe1 = (e1 * q).sum(1), torch.linalg.cross(e1, e0), torch.linalg.cross(e1, s)
    block = max(1, (1 << 24) // len(T))
    for i in range(0, n, block):
        r = d[i:i + block]
        det = r @ e1xe0.T
        inv = 1.0 / det
        u = (r @ sxe1.T) * inv
        w2 = (r @ q.T) * inv
        t = te1q * inv
        ok = (det.abs() > 0.0001) & (u >= 0) & (w2 >= 0) & (u + w2 <= 1) & (t > 0.001)
        t = torch.where(ok, t, torch.full_like(t, 1e30))
        t, k = t.min(1)
        near = t < best[i:i + block]
        bu, bv = u.gather(1, k[:, None]), w2.gather(1, k[:, None])
        g = at[0][k] * (1 - bu - bv) + at[1][k] * bu + at[2][k] * bv
        g = g / g.norm(dim=1, keepdim=True)
        normal[i:i + block] = torch.where(near[:, None], g, normal[i:i + block])
        hit[i:i + block] |= near
    film = torch.where(hit[:, None], (normal + 1) * 0.5, _sky64(sky, d))
    return {"film": film.reshape(h, w, 3).cpu().numpy(), "picked": None}


def _sky64(sky, d):
    """The Perez sky's colour of each direction."""
    r = sky.raw
    basis = torch.tensor([list(r.orthonormal_basis_u), list(r.orthonormal_basis_v), list(r.orthonormal_basis_w)],
                         dtype=torch.float64, device=d.device)
    e = d @ basis.T
    below = e[:, 2] < 0
    e = torch.cat([e[:, :2], e[:, 2:].clamp(min=0.001)], 1)
    e = e / e.norm(dim=1, keepdim=True)
    cos1 = e[:, 2].clamp(-1, 1)
    cosg = (e @ torch.tensor(list(r.sun_direction), dtype=torch.float64, device=d.device)).clamp(-1, 1)
    gamma, theta1, theta0 = torch.acos(cosg), torch.acos(cos1), r.theta

    def perez(c, zenith, theta_den):
        num = (1 + c[0] * torch.exp(c[1] / (cos1 + 0.01))) * (1 + c[2] * torch.exp(c[3] * gamma) + c[4] * cosg * cosg)
        den = (1 + c[0] * math.exp(c[1])) * (1 + c[2] * torch.exp(c[3] * theta_den) + c[4] * math.cos(theta0) ** 2)
        return zenith * num / den

    level = perez(r.perez_relative_luminance, r.zenith_relative_luminance, torch.full_like(theta1, theta0)) * 1e-4
    cx, cy = perez(r.perez_x, r.zenith_x, theta1), perez(r.perez_y, r.zenith_y, theta1)
    c0 = 1 / (0.0241 + 0.2562 * cx - 0.7341 * cy)
    c1, c2 = (-1.3515 - 1.7703 * cx + 5.9114 * cy) * c0, (0.03 - 31.4424 * cx + 30.0717 * cy) * c0
    X = 10246.121 + c1 * 187.75537 + c2 * 213.14803
    Y = 10676.695 + c1 * 192.59653 + c2 * 76.29494
    Z = 12372.504 + c1 * 3482.8765 + c2 * -235.71611
    xyz = torch.stack([X * level / Y, level, Z * level / Y], 1)
    to_rgb = torch.tensor([[3.2410042, -1.5373994, -0.49861607], [-0.9692241, 1.8759298, 0.041554242],
                           [0.05563942, -0.20401107, 1.0571486]], dtype=torch.float64, device=d.device)
    rgb = xyz @ to_rgb.T
    rgb = rgb + (-rgb.min(dim=1, keepdim=True).values).clamp(min=0)
    return torch.where(below[:, None], torch.full_like(rgb, 0.01), rgb)
