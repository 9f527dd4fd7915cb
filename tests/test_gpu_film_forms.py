"""The wide-filter film's two forms (a thread or a warp per output pixel) on
both sides of the line between them: films summed here, in numpy, from the
radiance of every path sample and its film position.  Box filters of other
radii weigh every sample by 1, and one tile holds the whole film, so a pixel is
the sum of the samples within the radius in raster and sample order: equal bit
for bit."""
import numpy as np
import pytest

from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu

U64 = np.uint64


def _mix64(x):
    x = x ^ (x >> U64(30))
    x = x * U64(0xbf58476d1ce4e5b9)
    x = x ^ (x >> U64(27))
    x = x * U64(0x94d049bb133111eb)
    return x ^ (x >> U64(31))


def _film_position(seed, pixel, sample):
    """The first two numbers of the path streams of (seed, pixel, sample): PCG32
    over the mixed seed and pixel, its 23 top bits as a float in [0, 1)."""
    mult = U64(0x5851f42d4c957f2d)
    inc = (sample.astype(U64) << U64(1)) | U64(1)
    state = (inc + _mix64((U64(seed) << U64(32)) ^ pixel.astype(U64))) * mult + inc
    out = []
    for _ in range(2):
        xs = ((((state >> U64(18)) ^ state) >> U64(27)) & U64(0xffffffff)).astype(np.uint32)
        rot = (state >> U64(59)).astype(np.uint32)
        u = (xs >> rot) | (xs << ((~rot + np.uint32(1)) & np.uint32(31)))
        out.append(((u >> np.uint32(9)) | np.uint32(0x3f800000)).view(np.float32) - np.float32(1))
        state = state * mult + inc
    return out


def _film(radiance, x, y, r, ov, step):
    """Every step-th pixel; radiance (H, W, spp, 3), film positions (H, W, spp)."""
    H, W, spp = x.shape
    yy, xx = np.mgrid[0:H:step, 0:W:step]
    film = np.zeros(xx.shape + (4,), np.float32)
    reach = int(np.ceil(r + 0.5))
    for dy in range(-reach, reach + 1):
        for dx in range(-reach, reach + 1):
            sy, sx = yy - ov + dy, xx - ov + dx
            ok = (sy >= 0) & (sy < H) & (sx >= 0) & (sx < W)
            cy, cx = np.clip(sy, 0, H - 1), np.clip(sx, 0, W - 1)
            for s in range(spp):
                # position on the screen, which starts ov pixels before the film
                px = (x[cy, cx, s] - np.float32(0.5)) - np.float32(-ov)
                py = (y[cy, cx, s] - np.float32(0.5)) - np.float32(-ov)
                m = ok & (xx >= np.ceil(px - r)) & (xx <= np.floor(px + r)) & (yy >= np.ceil(py - r)) & (yy <= np.floor(py + r))
                film[..., :3] += np.where(m[..., None], radiance[cy, cx, s], np.float32(0))
                film[..., 3] += m.astype(np.float32)
    return film


# (film, radius, samples): a warp per pixel where at least 96 samples reach the
# pixel's window on films below 97,280 pixels (640 per SM of 152), or 640 samples
# below 194,560; a pixel's window is 3x3 at radius 1, 5x5 at 1.6, 7x7 at 2.6
CASES = [((41, 33), 1.0, 10), ((41, 33), 1.0, 11), ((40, 40), 1.6, 4), ((330, 294), 1.0, 11), ((330, 295), 1.0, 11),
         ((331, 297), 2.6, 13), ((331, 297), 2.6, 14), ((450, 432), 2.6, 14), ((450, 433), 2.6, 14)]


@pytest.mark.parametrize("size,r,spp", CASES, ids=["%dx%d_r%g_%dspp" % (s + (r, n)) for s, r, n in CASES])
def test_wide_film_sums_the_samples_in_order(ctx, rtlib, size, r, spp):
    w, h = size
    s = scenes.cornell_box(w, h)
    s.camera["filter"] = D.box_filter(r, r)
    s.integrator = dict(s.integrator, max_depth=2)
    g = rtlib.Scene(ctx, s)
    pixel = np.repeat(np.arange(w * h), spp)
    sample = np.tile(np.arange(spp), w * h)
    try:
        film = g.render(spp, seed=9, block=512)
        rad = g.render_paths(pixel, sample, seed=9)
    finally:
        g.close()
    with np.errstate(over="ignore"):
        jx, jy = _film_position(9, pixel, sample)
    x = ((pixel % w).astype(np.float32) + jx).reshape(h, w, spp)
    y = ((pixel // w).astype(np.float32) + jy).reshape(h, w, spp)
    step = 1 if w < 100 else 5
    ref = _film(rad.reshape(h, w, spp, 3), x, y, np.float32(r), int(np.ceil(np.float32(r) - np.float32(0.5))), step)
    film = film[::step, ::step]
    assert np.array_equal(film[..., 3], ref[..., 3])
    assert np.array_equal(film[..., :3], ref[..., :3])
