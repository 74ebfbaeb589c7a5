"""Residency of the shade kernels of layered scenes: they wait on gathers, so a
register count that leaves one block per SM costs a fifth of the frame, which
no image shows."""
import pytest

from graph_kernels import kernels_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shades", [("pt", 1), ("bdpt", 2)])
def test_layered_shade_kernels_keep_two_blocks(rb, cuda, kind, shades):
    from renderbox2_b200.configs import CONFIG2 as C2
    from renderbox2_b200.render import (BidirectionalPathIntegratorLvcParams, BsdfLayer, DeviceScene, Integrator,
                                        PathIntegratorParams)
    torch = cuda
    scene = rb.RoomScene(seed=4, n_boxes=3, n_spheres=6, sphere_subdiv=1, n_lights=1, emission=10.0)
    layers = [[] if e.max() > 0 else [BsdfLayer("mirror" if i % 2 else "orennayar", tuple(float(x) for x in a))]
              for i, (a, e) in enumerate(zip(scene.albedo, scene.emission))]
    it = Integrator(rb.CudaTracer(rb.BVH(scene)), DeviceScene(scene, materials=layers))
    cam = rb.PerspectiveCamera(C2["eye"], C2["lookat"], C2["up"], (61, 34), C2["fov"])
    out = torch.empty((61 * 34, 3), device="cuda")
    pt = PathIntegratorParams(spp=1, max_depth=3)
    bd = BidirectionalPathIntegratorLvcParams(spp=1, max_path_length=4, connections=2)
    ks = kernels_of(torch, lambda: it.render_pt(cam, pt, out=out) if kind == "pt" else it.render_bdpt(cam, bd, out=out))
    found = {k["name"]: k for k in ks if "shade" in k["name"]}
    assert len(found) == shades
    for k in found.values():
        assert k["per_sm"] * k["block"] >= 512, k
