"""The shade kernels without the layered-material code against those with it: a
scene of single Lambertian layers is rendered as it is, with its materials set
as layers (still the plain kernels), and with one more material, a mirror that
no triangle has (the layered kernels, on the same surfaces).  Images are
bit-identical, for the path tracer, BDPT at one and several connections, and
the reference BDPT estimator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pt", "bdpt1", "bdpt3", "reference"])
def test_plain_and_layered_kernels_agree(rb, cuda, kind):
    from renderbox2_b200.configs import CONFIG2 as C2
    from renderbox2_b200.render import (BidirectionalPathIntegratorLvcParams, BsdfLayer, DeviceScene, Integrator,
                                        PathIntegratorParams)
    scene = rb.RoomScene(seed=4, n_boxes=3, n_spheres=12, sphere_subdiv=1, n_lights=2, emission=10.0)
    tracer = rb.CudaTracer(rb.BVH(scene))
    cam = rb.PerspectiveCamera(C2["eye"], C2["lookat"], C2["up"], (61, 34), C2["fov"])
    layers = [[] if e.max() > 0 else [BsdfLayer("lambertian", tuple(float(x) for x in a))]
              for a, e in zip(scene.albedo, scene.emission)]
    pad = np.zeros((1, 3), np.float32)
    more = dict(albedo=np.concatenate([scene.albedo, pad]), emission=np.concatenate([scene.emission, pad]))
    scenes = [DeviceScene(scene), DeviceScene(scene, materials=layers),
              DeviceScene(scene, materials=layers + [[BsdfLayer("mirror", (0.9, 0.9, 0.9))]], **more)]
    images = []
    for s in scenes:
        it = Integrator(tracer, s)
        if kind == "pt":
            images.append(it.render_pt(cam, PathIntegratorParams(spp=4, max_depth=6, seed=3)))
        elif kind == "reference":
            images.append(it.render_bdpt(cam, BidirectionalPathIntegratorLvcParams(
                spp=2, estimator="reference", num_prep_paths=200, connections=2, seed=3)))
        else:
            images.append(it.render_bdpt(cam, BidirectionalPathIntegratorLvcParams(
                spp=2, max_path_length=6, connections=int(kind[4:]), seed=3)))
    a, b, c = (x.cpu().numpy().view(np.uint32) for x in images)
    assert a.any() and np.array_equal(a, b) and np.array_equal(a, c)
