"""Wavefront stages at the ends of their range: no bounce, one, and the deepest
paths the entry points take.  Each frame is rendered as one wave and as one
sample per wave: images bit-identical (every sample is keyed on its own), ray
counts equal, primary rays one per sample, and no rays of a kind that the
depth leaves no room for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, SPP = 33, 17, 3


@pytest.fixture(scope="module")
def room(rb, cuda):
    from renderbox2_b200.configs import CONFIG2 as C2
    from renderbox2_b200.render import DeviceScene, Integrator
    scene = rb.RoomScene(seed=2, n_boxes=3, n_spheres=12, sphere_subdiv=1, n_lights=1, emission=10.0)
    tracer = rb.CudaTracer(rb.BVH(scene))
    cam = rb.PerspectiveCamera(C2["eye"], C2["lookat"], C2["up"], (W, H), C2["fov"])
    return tracer, Integrator(tracer, DeviceScene(scene)), cam


def both(it, render):
    got = []
    for paths in (0, W * H):
        it.set_wave(paths)
        got.append((render().cpu().numpy(), it.stats()))
    it.set_wave(0)
    (a, sa), (b, sb) = got
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and np.isfinite(a).all()
    counts = ("primary_rays", "extension_rays", "shadow_rays", "connection_rays", "light_rays")
    assert {k: sa[k] for k in counts} == {k: sb[k] for k in counts}
    assert sa["primary_rays"] == W * H * SPP
    return sa


@pytest.mark.parametrize("order", ["dfs", "cw8"])
@pytest.mark.parametrize("depth", [0, 1, 64])
def test_path_tracer_depths(rb, room, depth, order):
    from renderbox2_b200.render import PathIntegratorParams
    tracer, it, cam = room
    tracer.set_node_order(rb.NODE_ORDER_CW8 if order == "cw8" else rb.NODE_ORDER_DFS)
    st = both(it, lambda: it.render_pt(cam, PathIntegratorParams(spp=SPP, max_depth=depth, rr_start=60, seed=5)))
    assert 0 < st["shadow_rays"] <= (depth + 1) * W * H * SPP
    assert st["extension_rays"] <= depth * W * H * SPP and (depth == 0 or st["extension_rays"] > 0)


@pytest.mark.parametrize("order", ["dfs", "cw8"])
@pytest.mark.parametrize("length,connections", [(1, 1), (2, 2), (3, 8), (16, 1)])
def test_bdpt_lengths(rb, room, length, connections, order):
    from renderbox2_b200.render import BidirectionalPathIntegratorLvcParams
    tracer, it, cam = room
    tracer.set_node_order(rb.NODE_ORDER_CW8 if order == "cw8" else rb.NODE_ORDER_DFS)
    p = BidirectionalPathIntegratorLvcParams(spp=SPP, max_path_length=length, connections=connections, rr_start=14,
                                             seed=6)
    st = both(it, lambda: it.render_bdpt(cam, p))
    assert (st["light_rays"] > 0) == (length >= 3) and (st["connection_rays"] > 0) == (length >= 3)
    assert (st["shadow_rays"] > 0) == (length >= 2)


def test_bdpt_reference_deepest(rb, room):
    from renderbox2_b200.render import BidirectionalPathIntegratorLvcParams
    tracer, it, cam = room
    tracer.set_node_order(rb.NODE_ORDER_DFS)
    p = BidirectionalPathIntegratorLvcParams(spp=SPP, estimator="reference", num_prep_paths=100, connections=2,
                                             num_light_path_max_depth=16, num_cam_path_max_depth=63,
                                             cam_path_rrstart=60, seed=7)
    st = both(it, lambda: it.render_bdpt(cam, p))
    assert st["light_rays"] > 100 and st["connection_rays"] > 0
