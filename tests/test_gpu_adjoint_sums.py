"""GPU: the adjoint's sums. With more than 1,609 primitives a block's gradient entries do not fit its shared
memory, and every term goes to its entry in double precision. The scene shows it exactly: a plane fills the
image, paths end at their first hit, so the gradient of the plane's emission is the sum of the image weights -
whole numbers, half of them +-2^26, half from 1 to 7. Their sum is exact in double in any order, and loses
the small ones as soon as a few terms are added in float."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 2, 8])  # 1: the plain replay; 2 and 8: waves
def test_gradients_of_many_primitives_are_summed_in_double(spp):
    from dfpt import scene as sc
    from dfpt.diff import DiffRenderer
    from dfpt.kernel import RendererKernel

    b = sc.SceneBuilder()
    black = b.constant(0, 0, 0)
    grey = b.surface(sc.LAMBERTIAN, b.constant(0.5, 0.5, 0.5), black, black)
    b.primitive(b.plane((0, 0, 0), (1, 0, 0), (0, 1, 0)), grey)
    sphere = b.sphere((0, 0, 0), 0.1)
    for k in range(1700):  # behind the plane
        b.primitive(sphere, grey, position=(0.3 * (k % 40 - 20), 0.3 * (k // 40 - 20), -3.0))
    width, height = 96, 64
    b.camera((0, 0, 5), (0, 0, 0), 60.0, (width, height))
    params = dict(renderer_type=2, pt_ray_depth_maximum=1, pt_ray_depth_russian_roulette=5, tone_mapper_type=2)
    k = RendererKernel(b.compile("sums"), sc.SkyState((0.3, 0.5, 0.8), 2.0), params)
    k.update(width, height)
    d = DiffRenderer(k)
    d.forward(None, None, None, 2.0, (0.3, 0.5, 0.8), spp)
    rng = np.random.default_rng(spp)
    shape = (height, width, 3)
    weights = np.where(rng.random(shape) < 0.5, rng.choice([-2.0 ** 26, 2.0 ** 26], shape), rng.integers(1, 8, shape)).astype(np.float32)
    emission = d.backward(weights)["emission"]
    k.dispose()
    assert np.array_equal(emission[0], weights.astype(np.float64).sum((0, 1)))
    assert not emission[1:].any()


def test_kernel_set_switched_between_forward_and_backward():
    """The gradient rows belong to the forward; the backward's launches, whose grids follow the kernel set
    selected then, take no more blocks than there are rows. Gradients as without the switch: the replay is
    the same, pass by pass or in waves (rtol 1e-4 per group, what the order of float sums leaves there)."""
    from dfpt import synthetic
    from dfpt.diff import DiffRenderer
    from dfpt.kernel import RendererKernel
    from dfpt.scene import SkyState

    scene, params, (w, h), truth, start = synthetic.inverse_scene(seed=4, width=160, height=120, count=25)
    weights = np.random.default_rng(2).normal(size=(h, w, 3)).astype(np.float32)
    out = []
    for switched in (False, True):
        k = RendererKernel(scene, SkyState((0.3, 0.9, 0.25), 2.5), dict(params, seed=5))
        k.update(w, h)
        d = DiffRenderer(k)
        d.forward(start["albedo"], None, start["phong_exponent"], 2.5, (0.3, 0.9, 0.25), 4)
        k.set_strict(switched)
        out.append(d.backward(weights))
        k.dispose()
    for key in ("albedo", "emission", "phong_exponent", "sun_direction"):
        a, b = (np.asarray(g[key]).ravel() for g in out)
        assert np.linalg.norm(a) > 0
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(a), key
