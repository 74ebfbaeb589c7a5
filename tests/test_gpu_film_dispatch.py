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
