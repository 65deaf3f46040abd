"""GPU: terrain frames whose rays go to warps by place, at sizes around a launch's lanes (152 SMs x 4 blocks x 256 =
155,648), against the same pass through one tail launch, which takes its rays from the counter. Picked primitives
are equal; films differ in what the order of the sun rays' float sums leaves (rtol 1e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(1, 1), (33, 1), (201, 149), (608, 256), (397, 393), (641, 479)])
def test_terrain_frames_equal_the_tail_launch(width, height):
    from dfpt import scene as sc, synthetic
    from dfpt.kernel import RendererKernel

    b = sc.SceneBuilder()
    black, grey = b.constant(0, 0, 0), b.constant(0.5, 0.5, 0.5)
    surface = b.surface(sc.LAMBERTIAN, grey, black, black)
    b.primitive(b.terrain(0.5, 1.0, 0.0, 1.0, 8), surface)
    b.primitive(b.sphere((0, 0, 0), 1.0), surface, position=(0.0, 2.0, 0.0))
    b.camera((0, 2.0, 10.0), (0, 0, 0), 60.0, (width, height))
    scene = b.compile("terrain")
    _, sky, params, _ = synthetic.sphere_scene()
    out = []
    for tail in (-1, 0):
        k = RendererKernel(scene, sky, params)
        k.update(width, height)
        k.set_tuning("tail_bounce", tail)
        k.execute(1)
        film, samples = k.film()
        assert (samples == 1).all() and np.isfinite(film).all()
        out.append((film.copy(), k.primitive_offsets().copy()))
        k.dispose()
    assert np.array_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-5, atol=1e-6)
