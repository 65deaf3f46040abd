"""GPU: binned waves and binned plain passes give the film of unbinned passes, at sizes on both sides of
the binning grids' steps (the grids follow the slots of a launch) and of the one-block scan (up to
32,768 bins). Rays only change their order, so films agree to what float atomics leave (rtol 1e-5, as
for every pair of processing orders)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Bins of the wave (bounce rays, shadow rays): 768 and 64; 6,144 and 4,096; 49,152 and
# 32,768; 393,216 and 262,144.
@pytest.mark.parametrize("width,height,passes", [(37, 21, 2), (96, 64, 7), (256, 200, 9), (641, 479, 8)])
def test_binned_waves_equal_unbinned_passes(width, height, passes):
    from dfpt import synthetic
    from dfpt.kernel import RendererKernel
    from dfpt.scene import camera_set_resolution

    scene, sky, params, _ = synthetic.small_mesh_scene(width=width, height=height)
    camera_set_resolution(scene.camera, width, height)
    films = []
    for wide, binned in ((1, 0), (1, 1), (passes, 1)):
        k = RendererKernel(scene, sky, params)
        k.update(width, height)
        k.set_tuning("wide_samples", wide)
        k.set_tuning("pass_shadow_sort", binned)
        k.set_tuning("pass_ray_sort", 9 * binned)
        k.execute(passes)
        film, samples = k.film()
        assert (samples == passes).all()
        films.append((film.copy(), k.primitive_offsets().copy()))
        k.dispose()
    for film, picked in films[1:]:
        np.testing.assert_allclose(film, films[0][0], rtol=1e-5, atol=1e-6)
        assert np.array_equal(picked, films[0][1])
