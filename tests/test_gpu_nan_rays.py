"""Rays with NaN and infinite parts in the compressed 8-wide layout, against the
binary layout: equal records, and no walk of the whole tree for a ray whose
interval is not a number (it can hit nothing)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")


@pytest.fixture(scope="module")
def setup(rb, cuda):
    scene = rb.heightfield_for_triangles(1, 131840)
    return rb.CudaTracer(rb.BVH(scene)), rb.surface_rays(scene, 4, 256)[0]


def odd_rays(rays):
    """Every ordinary ray once with each odd value in tmin, tmax, both, and in the whole origin beside them."""
    out = []
    for lo, hi in ((NAN, None), (None, NAN), (NAN, NAN), (INF, None), (None, INF), (None, -INF), (-INF, None),
                   (-INF, INF), (INF, INF), (-INF, -INF)):
        for org in (None, NAN, INF, -INF):
            r = rays[:7].copy()
            if lo is not None:
                r[:, 3] = lo
            if hi is not None:
                r[:, 7] = hi
            if org is not None:
                r[:, :3] = org
            # A NaN or infinite origin with an interval of numbers walks every box in any layout.
            out.append(r if org is None or lo is NAN or hi is NAN else r[:1])
    return np.concatenate(out)


def test_records_equal_binary(rb, cuda, setup):
    torch = cuda
    tracer, rays = setup
    odd = torch.from_numpy(np.concatenate([odd_rays(rays), rays])).cuda()
    got = {}
    for order in (rb.NODE_ORDER_DFS, rb.NODE_ORDER_CW8):
        tracer.set_node_order(order)
        got[order] = [tracer.trace(odd), tracer.trace(odd, any_hit=True)[:, 0] >= 0, tracer.trace_occlusion(odd)]
    assert tracer.status() == 0
    for a, b in zip(*got.values()):
        assert a.equal(b)
    assert bool((got[rb.NODE_ORDER_CW8][0][-256:, 0] >= 0).any())


@pytest.mark.parametrize("lo,hi,org", [(NAN, None, NAN), (None, NAN, NAN), (NAN, NAN, None), (NAN, None, None)])
def test_no_walk_without_an_interval(rb, cuda, setup, lo, hi, org):
    torch = cuda
    tracer, rays = setup
    tracer.set_node_order(rb.NODE_ORDER_CW8)
    ray = rays[:1].copy()
    plain = torch.from_numpy(ray.copy()).cuda()
    if lo is not None:
        ray[:, 3] = lo
    if hi is not None:
        ray[:, 7] = hi
    if org is not None:
        ray[:, :3] = org
    odd, out = torch.from_numpy(ray).cuda(), torch.empty((1, 4), dtype=torch.int32, device="cuda")

    def ms(r):
        t = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            tracer.trace(r, out=out)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return sorted(t)[1]

    plain_ms, odd_ms = ms(plain), ms(odd)
    assert int(out[0, 0]) == -1
    assert odd_ms < 20 * plain_ms, (odd_ms, plain_ms)
