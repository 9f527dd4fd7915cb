"""The warp-per-pixel film of the wider reconstruction filters against the
oracle: radii on both sides of a whole number of pixels, sample counts on both
sides of a warp, ragged tiles."""
import numpy as np
import pytest

import oracle_lib as O
from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 5, 33])
@pytest.mark.parametrize("flt", [D.gaussian_filter(0.7, 0.49), D.gaussian_filter(1.0, 1.49), D.mitchell_filter(1.5, 1.51),
                                 D.gaussian_filter(2.0, 3.3), D.box_filter(2.5, 0.5)],
                         ids=["gauss_07_049", "gauss_10_149", "mitchell_15_151", "gauss_20_33", "box_25_05"])
def test_wide_film_matches_oracle(ctx, rtlib, flt, spp):
    s = scenes.cornell_box(37, 29)
    s.camera["filter"] = flt
    g = rtlib.Scene(ctx, s)
    try:
        film = g.render(spp, seed=3, block=12)
    finally:
        g.close()
    ref = O.OracleScene(s).render(spp, seed=3, block=12)
    assert np.array_equal(film[..., 3], ref[..., 3])   # the same weights summed in the same order
    err = np.abs(film[..., :3] - ref[..., :3]) / np.maximum(np.abs(ref[..., :3]), 1e-3)
    assert np.mean(err.max(-1) > 1e-3) <= 0.02   # paths whose branch flips on a last-ulp difference
