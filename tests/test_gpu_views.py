"""GPU: the per-pixel views at frame sizes on both sides of their launches' rules - a tile a warp or more, the
forms with 4 and with 8 resident blocks, more tiles than the launch has warps, widths and heights that are no
multiple of a tile's. The uncounted views (the packed pair walk or the walk of scenes without meshes, in tiles)
against the counting ones, which take rows: the picked primitives are equal, films to the rounding that two
compilations of the shading leave (rtol 1e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 152 SMs: 77,824 pixels fill 4 blocks per SM, 155,648 fill 8.
@pytest.mark.parametrize("width,height", [(3, 2), (41, 35), (319, 243), (320, 244), (641, 479)])
@pytest.mark.parametrize("kind", ["mesh", "spheres"])
def test_views_equal_counting_views(kind, width, height):
    from dfpt import synthetic
    from dfpt.kernel import RendererKernel
    from dfpt.scene import camera_set_resolution

    scene, sky, params = (synthetic.small_mesh_scene() if kind == "mesh" else synthetic.sphere_scene())[:3]
    scene.camera = camera_set_resolution(scene.camera.copy(), width, height)
    for renderer in (1, 3, 5, 6):
        out = []
        for counting in (False, True):
            k = RendererKernel(scene, sky, dict(params, renderer_type=renderer))
            k.update(width, height)
            k.set_counting(counting)
            k.execute(2)
            film, samples = k.film()
            assert (samples == 2).all()
            out.append((film.copy(), k.primitive_offsets().copy()))
            k.dispose()
        assert np.array_equal(out[0][1], out[1][1])
        np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-5, atol=1e-6)


def test_marcher_and_terrain_views_cover_the_frame():
    """Views that take rows from the work counter, at a size with more rows' pieces than warps: every pixel has
    its sample, and the marcher's image is the one that the launch without counting gives."""
    from dfpt import scene as sc, synthetic
    from dfpt.kernel import RendererKernel
    from dfpt.scene import camera_set_resolution

    width, height = 641, 479
    scene, sky, params = synthetic.sphere_scene()[:3]
    scene.camera = camera_set_resolution(scene.camera.copy(), width, height)
    images = []
    for counting in (False, True):
        k = RendererKernel(scene, sky, dict(params, renderer_type=4))
        k.update(width, height)
        k.set_counting(counting)
        k.execute(1)
        film, samples = k.film()
        assert (samples == 1).all()
        images.append(film.copy())
        k.dispose()
    assert np.array_equal(images[0], images[1])
    b = sc.SceneBuilder()
    black = b.constant(0, 0, 0)
    b.primitive(b.terrain(0.5, 1.0, 0.0, 1.0, 8), b.surface(sc.LAMBERTIAN, b.constant(0.5, 0.5, 0.5), black, black))
    b.camera((0, 2.0, 10.0), (0, 0, 0), 60.0, (width, height))
    k = RendererKernel(b.compile("terrain"), sky, dict(params, renderer_type=6))
    k.update(width, height)
    k.execute(1)
    film, samples = k.film()
    picked = k.primitive_offsets()
    k.dispose()
    assert (samples == 1).all() and np.isfinite(film).all()
    assert (picked == 0).any()
