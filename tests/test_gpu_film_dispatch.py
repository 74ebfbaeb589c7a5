"""Launches of the film's reconstruction: which kernel takes a film, in what
shape, and that images do not depend on it.  Bar for images: bit-identical to
the oracle's per-pixel sums (see test_gpu_film_strip)."""
import numpy as np
import pytest

from graph_kernels import kernels_of

pytestmark = pytest.mark.gpu


def samples(W, H, spp, seed=1):
    rng = np.random.Generator(np.random.PCG64(seed))
    pix = np.arange(W * H)
    base = np.tile(np.stack([pix % W, pix // W], 1).astype(np.float32), (spp, 1))
    xy = np.minimum(base + rng.uniform(0, 1, base.shape).astype(np.float32),
                    np.nextafter(base + 1, 0, dtype=np.float32)).astype(np.float32)
    return xy, rng.exponential(1.0, (spp * W * H, 4)).astype(np.float32)


def develop(torch, kind, xw, yw, W, H, spp, xy, L, out=None):
    from renderbox2_b200.render import Filter, film_develop
    return film_develop(Filter(kind, xw, yw, 2.0), W, H, spp, xy, L, out=out)


@pytest.mark.parametrize("W,H", [(256, 1), (257, 1), (701, 450)])
def test_gather_covers_the_film_in_one_pass(orc, cuda, W, H):
    """One block per 256 pixels: a grid that strides over the pixels leaves its last wave part empty."""
    torch = cuda
    xy, L = samples(W, H, 1)
    dxy, dL, out = torch.from_numpy(xy).cuda(), torch.from_numpy(L).cuda(), torch.empty((W * H, 3), device="cuda")
    (k,) = kernels_of(torch, lambda: develop(torch, "gaussian", 4.0, 4.0, W, H, 1, dxy, dL, out))
    assert "k_film_gather" in k["name"]
    assert k["grid"] == ((W * H + k["block"] - 1) // k["block"], 1, 1)
    want = orc.film("gaussian", 4.0, 4.0, 2.0, W, H, 1, xy, L)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_threads_develop_at_once(rb, orc, cuda, tmp_path):
    """Staged rows of 50 to 99 KB from several threads: the kernel's shared memory limit is one per device, so no
    thread may lower what another one's launch needs."""
    import ctypes as C
    import subprocess
    from pathlib import Path
    torch = cuda
    root = Path(__file__).resolve().parent.parent
    so = tmp_path / "film_threads.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-pthread", f"-I{root / 'include'}",
                    str(root / "tests" / "cpp" / "film_threads.cpp"), "-o", str(so)], check=True)

    class Job(C.Structure):
        _fields_ = [("kind", C.c_uint32), ("xw", C.c_float), ("yw", C.c_float), ("alpha", C.c_float),
                    ("w", C.c_uint32), ("h", C.c_uint32), ("spp", C.c_uint32), ("xy", C.c_void_p),
                    ("L", C.c_void_p), ("rgb", C.c_void_p), ("stream", C.c_void_p)]

    jobs, keep = (Job * 4)(), []
    for k, (W, H, spp) in enumerate([(33, 9, 79), (40, 5, 40), (64, 6, 60), (31, 8, 48)]):
        xy, L = samples(W, H, spp, seed=k)
        t = [torch.from_numpy(xy).cuda(), torch.from_numpy(L).cuda(), torch.empty((W * H, 3), device="cuda"),
             torch.cuda.Stream()]
        keep.append((t, orc.film("gaussian", 2.0, 2.0, 2.0, W, H, spp, xy, L)))
        jobs[k] = Job(3, 2.0, 2.0, 2.0, W, H, spp, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(),
                      t[3].cuda_stream)
    torch.cuda.synchronize()
    fn = C.CDLL(str(so)).film_threads
    develop_ptr = C.cast(rb.lib().rb2_film_develop, C.c_void_p)
    assert fn(develop_ptr, jobs, 4, 2000) == 0
    torch.cuda.synchronize()
    for t, want in keep:
        assert np.array_equal(t[2].cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("W,H,spp,xw,yw", [(33, 9, 40, 2.0, 2.0), (33, 9, 79, 2.0, 2.0), (33, 9, 80, 2.0, 2.0),
                                           (40, 9, 60, 3.0, 3.0), (40, 9, 62, 3.0, 3.0), (35, 5, 100, 1.0, 0.5)])
def test_large_staged_rows(orc, cuda, W, H, spp, xw, yw):
    """Around and above the 48 KB of shared memory that a launch gets without asking, up to the strip's limit."""
    torch = cuda
    xy, L = samples(W, H, spp, seed=spp)
    got = develop(torch, "gaussian", xw, yw, W, H, spp, torch.from_numpy(xy).cuda(), torch.from_numpy(L).cuda())
    want = orc.film("gaussian", xw, yw, 2.0, W, H, spp, xy, L)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("W,H,spp,xw,yw,strips", [
    (64, 64, 4, 3.0, 3.0, (2, 64, 1)),       # few strips: one row each
    (320, 180, 4, 3.0, 3.0, (10, 90, 1)),    # 8 warps per SM: two rows each
    (64, 64, 1, 3.0, 3.0, None), (480, 270, 1, 0.4, 2.0, None),  # one sample per pixel
    (33, 9, 178, 2.0, 2.0, (2, 9, 1)), (33, 9, 179, 2.0, 2.0, None),   # largest staged row
    (1000, 600, 12, 0.5, 0.5, None), (1000, 600, 12, 0.6, 0.6, (32, 75, 1))])  # share of the window in its rows
def test_route(orc, cuda, W, H, spp, xw, yw, strips):
    """The kernel and strip height that the measured rule picks on either side of its lines, with equal images."""
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    xy, L = samples(W, H, spp, seed=spp + W)
    dxy, dL, out = torch.from_numpy(xy).cuda(), torch.from_numpy(L).cuda(), torch.empty((W * H, 3), device="cuda")
    (k,) = kernels_of(torch, lambda: develop(torch, "triangle", xw, yw, W, H, spp, dxy, dL, out))
    assert ("k_film_strip" in k["name"]) == (strips is not None)
    if strips and sms == 148:
        assert k["grid"] == strips
    want = orc.film("triangle", xw, yw, 2.0, W, H, spp, xy, L)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
