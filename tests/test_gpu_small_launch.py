"""Small launches (a share of the rays per resident warp, no queue) against the
queue-driven kernel: the first n rays of a buffer traced alone give the records
of the whole buffer's launch, bit for bit, around the sizes where the share
changes (one ray, a warp, one and four rays per resident warp of 32 or 36 per
SM), in every layout and mode, with a stencil, and as batched jobs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOTAL = 60_000
SIZES = [1, 2, 31, 33, 4735, 4736, 4737, 5328, 5329, 18_943, 18_944, 18_945, 21_312, 21_313]


@pytest.fixture(scope="module")
def setup(rb, cuda):
    scene = rb.heightfield_scene(seed=5, grid_n=40, n_boxes=6)
    rays, _ = rb.surface_rays(scene, 9, TOTAL)
    mask = (np.random.default_rng(3).uniform(size=TOTAL) < 0.8).astype(np.uint8)
    return rb.CudaTracer(rb.BVH(scene)), cuda.from_numpy(rays).cuda(), cuda.from_numpy(mask).cuda()


@pytest.mark.parametrize("order", [0, 1, 2, 3])
def test_small_launch_equals_queue(setup, order):
    tracer, rays, mask = setup
    tracer.set_node_order(order)
    for m in (None, mask):
        closest, any_hit = tracer.trace(rays, stencil=m), tracer.trace(rays, any_hit=True, stencil=m)
        occ = tracer.trace_occlusion(rays, stencil=m)
        for n in SIZES:
            mn = None if m is None else m[:n]
            assert tracer.trace(rays[:n], stencil=mn).equal(closest[:n])
            assert tracer.trace(rays[:n], any_hit=True, stencil=mn).equal(any_hit[:n])
            assert tracer.trace_occlusion(rays[:n], stencil=mn).equal(occ[:n])
    assert tracer.status() == 0


@pytest.mark.parametrize("order,reorder", [(0, 0), (3, 0), (3, 4)])
def test_small_batches(rb, cuda, setup, order, reorder):
    torch = cuda
    tracer, rays, _ = setup
    tracer.set_node_order(order)
    closest, occ = tracer.trace(rays), tracer.trace_occlusion(rays)
    for sizes in ([1, 0, 3], [100, 1, 5000, 17], [18_000, 900, 40], [30_000, 7, 20_000]):
        jobs, want, at = [], [], 0
        for k, n in enumerate(sizes):
            mode = rb.MODE_CLOSEST if k % 2 == 0 else rb.MODE_OCCLUSION
            out = torch.full((n, 4), -7, dtype=torch.int32, device="cuda") if k % 2 == 0 else \
                torch.full((n,), 9, dtype=torch.uint8, device="cuda")
            jobs.append((tracer, rays[at:at + n], mode, out, None))
            want.append((closest if k % 2 == 0 else occ)[at:at + n])
            at += n
        b = rb.TraceBatch(jobs)
        b.set_config(node_order=order, reorder=reorder, chunk=4)
        s = torch.cuda.Stream()
        for capture in (False, True):
            if capture:
                b.capture(s)
            for _ in range(2):
                b.launch(s)
            s.synchronize()
            for (_, _, _, out, _), w in zip(jobs, want):
                assert out.equal(w)
                out.fill_(3)
        assert b.status() == 0


def test_small_isect(rb, cuda, setup):
    from renderbox2_b200.render import DeviceScene, trace_isect
    tracer, rays, mask = setup
    scene = DeviceScene(tracer_scene(rb))
    for order in (0, 3):
        tracer.set_node_order(order)
        full = trace_isect(tracer, scene, rays, any_hit=False, stencil=mask)
        for n in (1, 33, 4737, 18_945):
            part = trace_isect(tracer, scene, rays[:n], any_hit=False, stencil=mask[:n])
            for k, x in part.t.items():
                w = full[k][..., :n] if k in part.VEC else full[k][:n]
                assert x.nan_to_num(nan=-5).equal(w.nan_to_num(nan=-5)) if x.is_floating_point() else x.equal(w)


def tracer_scene(rb):
    return rb.heightfield_scene(seed=5, grid_n=40, n_boxes=6)
