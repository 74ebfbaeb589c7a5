"""What a caller's launch configuration does to small launches (at most four rays
per resident warp): ctas_per_sm limits the grid, with unchanged records, and
the autotuner does not search shapes that such launches do not have."""
import pytest

from graph_kernels import kernels_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(rb, cuda):
    scene = rb.heightfield_scene(seed=5, grid_n=40, n_boxes=6)
    rays, _ = rb.surface_rays(scene, 9, 20_000)
    return rb.CudaTracer(rb.BVH(scene)), cuda.from_numpy(rays).cuda()


@pytest.mark.parametrize("order", [0, 2, 3])
@pytest.mark.parametrize("block,ctas", [(64, 1), (64, 2), (64, 3), (128, 1), (0, 2), (256, 1), (256, 2), (256, 16)])
def test_cta_limit_holds(rb, cuda, setup, order, block, ctas):
    torch = cuda
    tracer, rays = setup
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tracer.set_node_order(order)
    tracer.set_launch()
    want = tracer.trace(rays)
    try:
        tracer.set_launch(ctas_per_sm=ctas, block_threads=block)
        for n in (1, 33, 147, 592, 593, 2368, 2369, 18_944, 20_000):
            out = torch.empty((n, 4), dtype=torch.int32, device="cuda")
            (k,) = kernels_of(torch, lambda: tracer.trace(rays[:n], out=out))
            assert k["grid"][0] * k["block"] <= sms * ctas * (block or 128), (n, k)
            assert out.equal(want[:n])
    finally:
        tracer.set_launch()
    assert tracer.status() == 0


def test_batch_cta_limit_and_autotune(rb, cuda, setup):
    torch = cuda
    tracer, rays = setup
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tracer.set_node_order(0)
    want = tracer.trace(rays[:3000])
    out = torch.empty((3000, 4), dtype=torch.int32, device="cuda")
    b = rb.TraceBatch([(tracer, rays[:1000], rb.MODE_CLOSEST, out[:1000], None),
                       (tracer, rays[1000:3000], rb.MODE_CLOSEST, out[1000:], None)])
    b.set_config(ctas_per_sm=1, block_threads=128)
    ks = kernels_of(torch, lambda: b.launch())
    assert max(k["grid"][0] * k["block"] for k in ks) <= sms * 128
    torch.cuda.synchronize()
    assert out.equal(want)
    cfg, _ = b.autotune(torch.cuda.Stream(), reps=1)
    assert (cfg["block_threads"], cfg["regs"], cfg["chunk"]) == (128, 64, 1)
