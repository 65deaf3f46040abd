"""GPU: the packed pair walk keeps the hit that the reference's preorder keeps where triangles meet.

Rays along an edge that two triangles share hit both at the same distance, or at distances an ulp apart, and
often meet the second one's box exactly at the hit: which triangle is kept then depends on the order of the
walk. The mesh here has its vertices on the rays of every other pixel, at varying depth, so that the rays of
every other column and row run along edges and through vertices, to the left and to the right of the camera's
axis. Hits of uncounted walks (the packed pair walk) equal those of counting walks (the threaded and compact
walks, in preorder) bit for bit: triangles, distances and normals, in both kernel sets.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _builder(width, height):
    from dfpt import scene as sc

    b = sc.SceneBuilder()
    black = b.constant(0, 0, 0)
    b.primitive(b.plane((0, -3, 0), (0, -3, 1), (1, -3, 0)), b.surface(sc.LAMBERTIAN, b.constant(0.5, 0.5, 0.5), black, black))
    b.camera((0.3, 0.7, 6.0), (0.3, 0.7, 0.0), 60.0, (width, height))
    return b, black


def _edges_on_rays(width, height, flat):
    from dfpt import scene as sc, synthetic

    c = _builder(width, height)[0].compile("camera").camera.astype(np.float64)
    eye, u, v, w = c[1:4], c[7:10], c[10:13], c[13:16]
    fx, fy = np.tan(np.radians(c[4]) / 2), np.tan(np.radians(-c[5]) / 2)
    xs, ys = np.arange(0, width, 2), np.arange(0, height, 2)
    sx, sy = 2 * (xs + 0.5) / (c[16] - 1) - 1, 2 * (ys + 0.5) / (c[17] - 1) - 1
    depth = np.random.default_rng(width).uniform(4.0, 6.0, (len(ys), len(xs)))
    if flat:
        depth[:] = 5.0  # every box flat in the viewing direction
    direction = w + u * (fx * sx)[None, :, None] + v * (fy * sy)[:, None, None]
    positions = (eye + depth[:, :, None] * direction).reshape(-1, 3)
    n = len(xs)
    quads = [(j * n + i, j * n + i + 1, (j + 1) * n + i + 1, (j + 1) * n + i) for j in range(len(ys) - 1) for i in range(n - 1)]
    indices = np.asarray([t for p, q, r, s in quads for t in ((p, q, r), (p, r, s))], np.int32)
    b, black = _builder(width, height)
    normals = synthetic.vertex_normals(positions, indices)
    mesh = b.mesh(positions, indices, normals, np.zeros((len(positions), 2)), synthetic.tangents_for(normals))
    b.primitive(mesh, b.surface(sc.LAMBERTIAN, b.constant(0.7, 0.6, 0.5), black, black))
    params = dict(renderer_type=2, pt_ray_depth_maximum=3, pt_ray_depth_russian_roulette=3, tone_mapper_type=2)
    return b.compile("edges"), sc.SkyState((0.5, 0.7, 0.4), 2.5), params


def _hits(scene, sky, params, width, height, counting):
    from dfpt.kernel import RendererKernel

    k = RendererKernel(scene, sky, params)
    k.update(width, height)
    k.set_record_hits(True)
    k.set_counting(counting)
    k.execute(1)
    out = [a.copy() for a in k.hits()]
    k.dispose()
    return out


@pytest.mark.parametrize("width,height,flat", [(72, 56, False), (203, 151, False), (640, 360, False), (203, 151, True)])
def test_rays_along_shared_edges_keep_the_preorder_hit(width, height, flat):
    scene, sky, params = _edges_on_rays(width, height, flat)
    for renderer in (1, 2, 3, 5, 6):
        uncounted, counted = (_hits(scene, sky, dict(params, renderer_type=renderer), width, height, c) for c in (False, True))
        assert (counted[2] >= 0).sum() > width * height // 2, "the mesh does not fill the image"
        for a, b in zip(uncounted, counted):
            assert np.array_equal(a, b), (renderer, int((np.asarray(a) != np.asarray(b)).sum()))


def _skipped_parent(lefts, chain):
    """A mesh tree in which a skipped node names the node that a chain of `chain` left children hangs from its
    child, `lefts` + 1 levels above that node's place in the walk's tree."""
    from dfpt import scene as sc, synthetic

    count = lefts + chain + 3
    corners = []
    for k in range(count):
        z, s = 0.02 * k, 2.0 * (1.0 - k / (count + 10.0))
        corners += [(-s + 0.3, -s + 0.7, z), (s + 0.3, -0.8 * s + 0.7, z), (0.1 * s + 0.3, s + 0.7, z - 0.05)]
    b, black = _builder(72, 56)
    positions, indices = np.asarray(corners), np.arange(3 * count, dtype=np.int32).reshape(-1, 3)
    normals = synthetic.vertex_normals(positions, indices)
    mesh = b.mesh(positions, indices, normals, np.zeros((len(positions), 2)), synthetic.tangents_for(normals))
    b.primitive(mesh, b.surface(sc.LAMBERTIAN, b.constant(0.7, 0.6, 0.5), black, black))
    scene = b.compile("skipped")
    point = scene.point3fs.reshape(-1)
    tris = np.arange(0, scene.triangles.size, 12)
    tri_corners = np.stack([[point[scene.triangles[t + v]:scene.triangles[t + v] + 3] for v in range(3)] for t in tris])
    lo, hi = tri_corners.min((0, 1)) - 0.1, tri_corners.max((0, 1)) + 0.1  # one box for every node
    box = [point.size, point.size + 3]
    # Nodes in order: (kind, name, next name). Inner nodes' left child is the node behind them.
    nodes = [("inner", f"i{k}", f"r{k - 1}" if k else None) for k in range(lefts)]
    after = f"r{lefts - 1}"
    nodes += [("inner", "top", after), ("leaf", "a", "x0"), ("inner", "skipped", after), ("leaf", "o", "x0")]
    nodes += [("inner", f"x{k}", f"y{k - 1}" if k else after) for k in range(chain)]
    nodes += [("leaf", "bottom", f"y{chain - 1}")] + [("leaf", f"y{k}", f"y{k - 1}" if k else after) for k in reversed(range(chain))]
    nodes += [("leaf", f"r{k}", f"r{k - 1}" if k else None) for k in reversed(range(lefts))]
    at, offsets = 0, {}
    for kind, name, _ in nodes:
        offsets[name] = at
        at += 5 if kind == "inner" else 6
    out, tri = [], iter(tris)
    for kind, name, following in nodes:
        nxt = -1 if following is None else offsets[following]
        out += [1, nxt, *box, offsets[name] + 5] if kind == "inner" else [2, nxt, *box, 1, int(next(tri))]
    scene.primitives[3 + 1] = scene.bounding_volume_hierarchies.size
    scene.bounding_volume_hierarchies = np.concatenate([scene.bounding_volume_hierarchies, np.asarray(out, np.int32)])
    scene.point3fs = np.concatenate([point, lo, hi]).astype(np.float32)
    params = dict(renderer_type=2, pt_ray_depth_maximum=3, pt_ray_depth_russian_roulette=3, tone_mapper_type=2)
    return scene, sc.SkyState((0.5, 0.7, 0.4), 2.5), params


@pytest.mark.parametrize("lefts,chain", [(3, 5), (10, 53), (10, 60), (40, 60)])
def test_depth_of_trees_with_skipped_nodes(lefts, chain):
    """A ray through every box has an entry pending per level: trees deeper than the stack keep another walk."""
    scene, sky, params = _skipped_parent(lefts, chain)
    for renderer in (1, 2, 3):
        uncounted, counted = (_hits(scene, sky, dict(params, renderer_type=renderer), 72, 56, c) for c in (False, True))
        assert (counted[2] >= 0).any()
        for a, b in zip(uncounted, counted):
            assert np.array_equal(a, b)
