"""The film's strip gather at the edges of its tiling: images narrower and
wider than a strip, one row, more rows than a strip, half-widths that reach 1,
2 and 3 rows and the wider ones and larger sample counts that the per-pixel
gather keeps.  Bar: bit-identical to the oracle's per-pixel sums, which add
the same products in the same order; an infinite sample reaches only the
pixels of its window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,spp,kind,xw,yw", [
    (1, 1, 1, "gaussian", 2.0, 2.0), (31, 1, 3, "triangle", 2.0, 0.5), (33, 7, 2, "gaussian", 0.5, 2.0),
    (64, 70, 1, "box", 0.5, 0.5), (65, 130, 4, "gaussian", 2.0, 2.0), (40, 9, 17, "triangle", 1.7, 2.49),
    (37, 11, 5, "gaussian", 3.1, 1.0), (20, 30, 2, "gaussian", 2.5, 3.0), (20, 12, 3, "box", 4.2, 6.0),
    (12, 10, 90, "gaussian", 2.0, 2.0), (12, 10, 300, "triangle", 2.0, 2.0), (200, 3, 6, "gaussian", 9.0, 2.0)])
def test_strip_gather_equals_oracle(rb, orc, cuda, W, H, spp, kind, xw, yw):
    from renderbox2_b200.render import Filter, film_develop
    torch = cuda
    rng = np.random.Generator(np.random.PCG64(W * H + spp))
    pix = np.arange(W * H)
    base = np.tile(np.stack([pix % W, pix // W], 1).astype(np.float32), (spp, 1))
    frac = rng.uniform(0, 1, base.shape).astype(np.float32)
    frac[rng.uniform(size=frac.shape) < 0.05] = 0.0   # on pixel edges
    frac[rng.uniform(size=frac.shape) < 0.05] = 0.5   # at pixel centres
    xy = np.minimum(base + frac, np.nextafter(base + 1, 0, dtype=np.float32)).astype(np.float32)
    L = rng.exponential(1.0, (spp * W * H, 4)).astype(np.float32)
    L[0, 0] = np.inf
    with np.errstate(invalid="ignore", over="ignore"):
        want = orc.film(kind, xw, yw, 2.0, W, H, spp, xy, L)
    got = film_develop(Filter(kind, xw, yw, 2.0), W, H, spp, torch.from_numpy(xy).cuda(),
                       torch.from_numpy(L).cuda()).cpu().numpy()
    assert np.array_equal(np.isinf(got), np.isinf(want)) and np.array_equal(np.isnan(got), np.isnan(want))
    fine = np.isfinite(want)
    assert np.array_equal(got[fine].view(np.uint32), want[fine].view(np.uint32))
