"""Batches at the ends of what rb2_batch_create takes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_jobs", [0, 1, 3])
@pytest.mark.parametrize("order", [0, 3])
def test_batch_without_rays(rb, cuda, n_jobs, order):
    """Jobs that hold no ray, or no job at all: every call works and nothing is written."""
    torch = cuda
    tracer = rb.CudaTracer(rb.BVH(rb.heightfield_scene(seed=5, grid_n=8, n_boxes=2)))
    out = torch.full((4, 4), 7, dtype=torch.int32, device="cuda")
    rays = torch.zeros((0, 8), device="cuda")
    b = rb.TraceBatch([(tracer, rays, rb.MODE_CLOSEST, out, None)] * n_jobs)
    b.set_config(node_order=order)
    s = torch.cuda.Stream()
    b.launch(s)
    b.capture(s)
    b.launch(s)
    cfg, ms = b.autotune(s, reps=1)
    assert cfg["node_order"] in (0, 1, 2, 3) and ms >= 0.0
    b.capture(s)
    b.launch(s)
    s.synchronize()
    assert b.status() == 0 and bool((out == 7).all())
