"""GPU: batches in which every scene has a terrain (their launches fill the warps) and batches in which some have
one, at sizes on both sides of a launch's warps, against the same scenes rendered one by one. Samples and their
random streams are the same; films differ in what the order of the sun rays' float sums leaves (rtol 1e-5, as
the other batch tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp", [(7, 5, 1), (97, 61, 3), (321, 243, 2)])
@pytest.mark.parametrize("kinds", ["tt", "ts"])
def test_terrain_batches_equal_single_renders(kinds, width, height, spp):
    from dfpt import scene as sc, synthetic
    from dfpt.batch import BatchRenderer
    from dfpt.kernel import RendererKernel

    b = sc.SceneBuilder()
    black, grey = b.constant(0, 0, 0), b.constant(0.5, 0.5, 0.5)
    surface = b.surface(sc.LAMBERTIAN, grey, black, black)
    b.primitive(b.terrain(0.5, 1.0, 0.0, 1.0, 8), surface)
    b.primitive(b.sphere((0, 0, 0), 1.0), surface, position=(0.0, 2.0, 0.0))
    b.camera((0, 2.0, 10.0), (0, 0, 0), 60.0, (width, height))
    spheres, sky, params, _ = synthetic.sphere_scene(width=width, height=height)
    scenes = [b.compile("terrain") if kind == "t" else spheres for kind in kinds]
    batch = BatchRenderer()
    for scene in scenes:
        batch.add(scene, width, height, spp, sky, params)
    batch.render()
    for index, scene in enumerate(scenes):
        film, samples = batch.film(index)
        k = RendererKernel(scene, sky, params)
        k.update(width, height)
        k.execute(spp)
        alone, alone_samples = k.film()
        k.dispose()
        assert np.array_equal(samples, alone_samples) and (samples == spp).all()
        np.testing.assert_allclose(film, alone, rtol=1e-5, atol=1e-6)
    batch.dispose()
