"""GPU: the packed pair walk (what configurations 16 and 17 and the per-pixel modes run when nothing
is counted) against the counting walks of the same build, which follow the reference's preorder.

The ray caster's kernels keep the reference's order in both, so hits and bytes are equal; the path
tracer's films agree to the rounding that float atomics leave (rtol 1e-5, as for every other pair
of walk orders). Trees at the edges: a root that is a leaf, two leaves, chains of boxes deep enough
to leave the shared-memory stack, as deep as the walk takes and one level deeper, boxes that do not nest (the scene
then keeps the counting walk's order), meshes with shared and with different matrices, every
culling mode. Scenes without meshes take a walk of their own (the culling BVH nearer child first): from
no bounded primitive to 90, spheres and triangles, and pairs of them in the same place.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh_scene(positions, indices, copies=1, spread=0.0, seed=0):
    """`copies` primitives of one mesh on a plane; spread 0: all with the same matrix."""
    from dfpt import scene as sc, synthetic

    rng = np.random.default_rng(seed)
    b = sc.SceneBuilder()
    black = b.constant(0, 0, 0)
    b.primitive(b.plane((0, -3, 0), (0, -3, 1), (1, -3, 0)), b.surface(sc.LAMBERTIAN, b.constant(0.5, 0.5, 0.5), black, black))
    positions = np.asarray(positions, np.float64)
    indices = np.asarray(indices, np.int32).reshape(-1, 3)
    n = synthetic.vertex_normals(positions, indices)
    mesh = b.mesh(positions, indices, n, np.zeros((len(positions), 2)), synthetic.tangents_for(n))
    for k in range(copies):
        surf = b.surface((sc.LAMBERTIAN, sc.PHONG, sc.REFLECTION)[k % 3], b.constant(*rng.uniform(0.3, 0.9, 3)), black, black)
        offset = rng.uniform(-spread, spread, 3) if spread else np.zeros(3)
        b.primitive(mesh, surf, position=tuple(float(v) for v in offset), scale=(1.0 + 0.1 * k * bool(spread),) * 3)
    b.camera((0.3, 0.7, 6.0), (0.05, 0.0, 0.0), 60.0, (72, 56))
    params = dict(renderer_type=2, pt_ray_depth_maximum=5, pt_ray_depth_russian_roulette=3, tone_mapper_type=2)
    return b.compile("walk"), sc.SkyState((0.5, 0.7, 0.4), 2.5), params


def _triangles(count):
    """`count` triangles facing the camera, the nearer ones smaller."""
    v = []
    for k in range(count):
        z, s = 0.02 * k, 2.0 * (1.0 - k / 80.0)
        v += [(-s + 0.013 * k, -s, z), (s, -0.8 * s, z), (0.1 * s + 0.01 * k, s, z - 0.05)]
    return v, np.arange(3 * count)


def _chain(compiled):
    """The mesh's tree as a chain: every inner node's left child holds all but one of its triangles,
    the right one that one, so a ray through all of them has an entry pending per level."""
    prim = 3  # the mesh's place in the primitives array (behind the plane)
    tris = np.arange(0, compiled.triangles.size, 12)
    count = len(tris)
    p = compiled.point3fs.reshape(-1)
    corners = np.stack([[p[compiled.triangles[t + v]:compiled.triangles[t + v] + 3] for v in range(3)] for t in tris])
    boxes, nodes = [], []

    def box(first, last):  # triangles first .. last - 1
        c = corners[first:last].reshape(-1, 3)
        boxes.extend([c.min(0), c.max(0)])
        at = p.size + 3 * (len(boxes) - 2)
        return [at, at + 3]

    # Preorder: the chain of inner nodes over 0 .. n - 1, n = count .. 2, then the leaves 0, 1, .. count - 1.
    inner, leaf = 5 * (count - 1), 6
    for n in range(count, 1, -1):
        at = 5 * (count - n)
        after = inner + leaf * n if n < count else -1  # what follows the node's last leaf (n - 1)
        nodes += [1, after, *box(0, n), at + 5]
    for k in range(count):
        nodes += [2, inner + leaf * (k + 1) if k + 1 < count else -1, *box(k, k + 1), 1, int(tris[k])]
    root = compiled.bounding_volume_hierarchies.size
    compiled.bounding_volume_hierarchies = np.concatenate([compiled.bounding_volume_hierarchies, np.asarray(nodes, np.int32)])
    compiled.point3fs = np.concatenate([p, np.asarray(boxes, np.float32).reshape(-1)])
    compiled.primitives[prim + 1] = root
    return compiled


def _flat_scene(count, shape, duplicates=False):
    """`count` spheres or triangle primitives over a plane and no mesh; duplicates: every second one
    where the one before it is, with another material (equal distances: the first one counts)."""
    from dfpt import scene as sc, synthetic

    rng = np.random.default_rng(count)
    b = sc.SceneBuilder()
    black = b.constant(0, 0, 0)
    b.primitive(b.plane((0, -1.5, 0), (0, -1.5, 1), (1, -1.5, 0)), b.surface(sc.LAMBERTIAN, b.constant(0.5, 0.5, 0.5), black, black))
    sphere = b.sphere((0, 0, 0), 0.35)
    position = np.zeros(3)
    for k in range(count):
        if not (duplicates and k % 2):
            position = rng.uniform((-2.5, -1.5, -3.0), (2.5, 1.8, 1.5))
        surf = b.surface((sc.LAMBERTIAN, sc.GLASS, sc.PHONG, sc.CLEAR_COAT)[k % 4], b.constant(*rng.uniform(0.3, 0.9, 3)), black, black)
        if shape == "sphere":
            b.primitive(sphere, surf, position=tuple(float(v) for v in position))
        else:
            v = position + np.asarray([(0.0, 0.5, 0.0), (-0.5, -0.3, 0.1), (0.5, -0.4, -0.2)])
            n = synthetic.vertex_normals(v, np.arange(3).reshape(1, 3))
            b.primitive(b.mesh(v, [[0, 1, 2]], n, np.zeros((3, 2)), synthetic.tangents_for(n), as_mesh=False), surf)
    b.camera((0.3, 0.7, 6.0), (0.05, 0.0, 0.0), 60.0, (72, 56))
    return b.compile("flat"), sc.SkyState((0.5, 0.7, 0.4), 2.5), dict(renderer_type=2, pt_ray_depth_maximum=5, pt_ray_depth_russian_roulette=3, tone_mapper_type=2)


def _scene(name):
    from dfpt import synthetic

    if name.startswith("flat_"):
        _, shape, count = name.split("_")[:3]
        return _flat_scene(int(count), shape, name.endswith("twice"))
    if name == "sphere":
        pos, idx, _, _, _ = synthetic.displaced_icosphere(6, 0.2, 4, radius=1.7)
        return _mesh_scene(pos, idx)
    if name in ("shared_matrix", "own_matrices", "many", "crowd"):
        # A ray through the crowd enters up to 70 boxes, more than a round of 16 candidates.
        pos, idx, _, _, _ = synthetic.displaced_icosphere(3, 0.2, 4, radius=0.9 if name != "crowd" else 0.3)
        copies, spread = {"shared_matrix": (4, 0.0), "own_matrices": (4, 1.8), "many": (12, 1.8), "crowd": (70, 0.9)}[name]
        return _mesh_scene(pos, idx, copies=copies, spread=spread)
    count = {"one": 1, "two": 2, "five": 5, "chain": 40, "deepest": 65, "too_deep": 66, "not_nested": 9}[name]
    compiled, sky, params = _mesh_scene(*_triangles(count))
    if name in ("chain", "deepest", "too_deep"):
        compiled = _chain(compiled)
    if name == "not_nested":
        bvh, p = compiled.bounding_volume_hierarchies, compiled.point3fs
        root = int(compiled.primitives[3 + 1])  # the mesh primitive's tree: {type, next, min, max, left}
        assert bvh[root] == 1
        p[int(bvh[root + 3]) + 2] -= np.float32(0.4)  # the root ends before its nearest triangle
    return compiled, sky, params


def _render(compiled, sky, params, counting, culling, passes):
    from dfpt.kernel import RendererKernel

    k = RendererKernel(compiled, sky, params)
    k.update(72, 56)
    k.set_tuning("primitive_culling", culling)
    k.set_record_hits(passes == 1)
    k.set_counting(counting)
    k.execute(passes)
    out = [k.film()[0].copy(), k.get().copy(), k.primitive_offsets().copy()]
    if passes == 1:
        out += [a.copy() for a in k.hits()]
    k.dispose()
    return out


@pytest.mark.parametrize("name", ["one", "two", "five", "sphere", "chain", "deepest", "too_deep", "not_nested", "shared_matrix", "own_matrices", "many", "crowd",
                                  "flat_sphere_0", "flat_sphere_3", "flat_sphere_8", "flat_sphere_90", "flat_sphere_90_twice", "flat_triangle_30",
                                  "flat_triangle_30_twice"])
def test_packed_walk_equals_counting_walk(name):
    compiled, sky, params = _scene(name)
    for culling in ((0, 1, 2) if compiled.primitive_count > 8 else (0,)):
        for renderer in (3, 1, 5, 6):
            a, b = (_render(compiled, sky, dict(params, renderer_type=renderer), c, culling, 1) for c in (False, True))
            assert (a[3] >= 0).any(), "no ray hits the scene"
            if renderer == 3:
                for x, y in zip(a, b):
                    assert np.array_equal(x, y), (name, culling)
            else:
                assert np.array_equal(a[2], b[2])
                np.testing.assert_allclose(a[0], b[0], rtol=1e-5, atol=1e-6)
        for passes in (1, 3):
            a, b = (_render(compiled, sky, params, c, culling, passes) for c in (False, True))
            assert np.array_equal(a[2], b[2])
            np.testing.assert_allclose(a[0], b[0], rtol=1e-5, atol=1e-6)


def test_transform_update_changes_the_matrix_runs():
    """dfpt_set_transforms on meshes that shared one matrix: the walk's runs follow."""
    from dfpt.kernel import RendererKernel

    compiled, sky, params = _scene("shared_matrix")
    moved_o = compiled.primitives_object_to_world.reshape(-1, 16).copy()
    moved_w = compiled.primitives_world_to_object.reshape(-1, 16).copy()
    for i, dx in ((2, 1.3), (4, -1.1)):
        moved_o[i, 3] += dx
        moved_w[i, 3] -= dx
    films = []
    for counting in (False, True):
        k = RendererKernel(compiled.copy(), sky, dict(params, renderer_type=3))
        k.update(72, 56)
        k.set_record_hits(True)
        k.set_counting(counting)
        k.execute(1)
        before = k.hits()[0].copy()
        k.compiled.primitives_object_to_world = moved_o.reshape(-1).astype(np.float32)
        k.compiled.primitives_world_to_object = moved_w.reshape(-1).astype(np.float32)
        k.update_primitives()
        k.execute(1)
        films.append([before] + [a.copy() for a in k.hits()])
        k.dispose()
    assert not np.array_equal(films[0][0], films[0][1])
    for x, y in zip(*films):
        assert np.array_equal(x, y)
