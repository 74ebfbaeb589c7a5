"""The compressed 8-wide layout where its box arithmetic rounds most: small
triangles far from the origin (a node's biased origin, origin less 32768 cells,
is rounded to a float there), and rays from up to 100 times the scene's
largest coordinate.  Its boxes contain the binary layout's with a margin for
that rounding, so no ray may find less than it finds there; a closest hit may
only be nearer (a triangle whose exact box the binary slab test rounded away)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset,size,reach", [((1000.0, -2000.0, 1500.0), 0.02, 0.0), ((0.0, 0.0, 4096.0), 0.3, 0.0),
                                               ((1.0e6, 1.0e6, -1.0e6), 40.0, 0.0), ((30.0, 20.0, 10.0), 0.02, 100.0),
                                               ((1.0e-6, 0.0, 0.0), 1.0e-3, 100.0)])
def test_nothing_is_lost(rb, cuda, offset, size, reach):
    torch = cuda
    rng = np.random.Generator(np.random.PCG64(11))
    n, off = 20_000, np.array(offset)
    centre = rng.uniform(-50 * size, 50 * size, (n, 1, 3)) + off
    v = (centre + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32)
    scene = rb.Scene().add_mesh(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))
    tracer = rb.CudaTracer(rb.BVH(scene))
    m = 50_000
    target = v[rng.integers(0, n, m)].mean(1).astype(np.float64)
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[: m // 10, 0] = 0.0   # in planes of the boxes' axes, and along one
    d[: m // 20, 1] = 0.0
    far = rng.uniform(0.5, 1.0, (m, 1)) * reach * np.abs(v).max()
    dist = far if reach else rng.uniform(1, 60, (m, 1)) * size
    rays = np.zeros((m, 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = target - d * dist, d, 3.0e38
    rays = torch.from_numpy(rays).cuda()
    tracer.set_node_order(rb.NODE_ORDER_DFS)
    want = tracer.trace(rays)
    tracer.set_node_order(rb.NODE_ORDER_CW8)
    got, occ = tracer.trace(rays), tracer.trace_occlusion(rays)
    hit, t, t_bin = want[:, 0] >= 0, got[:, 1].view(torch.float32), want[:, 1].view(torch.float32)
    assert int(hit.sum()) > m // 4
    assert bool((got[hit, 0] >= 0).all()) and bool((occ[hit] == 1).all())
    assert bool((t[hit] <= t_bin[hit]).all())
    assert float((t[hit] == t_bin[hit]).float().mean()) > 0.99
    assert tracer.status() == 0
