"""The tile-order table written on the device (k_tile_orders): films of ragged
sizes and block shapes against the oracle's, whose job grid is the reference's
(a block larger than the film, one pixel, single rows and columns)."""
import numpy as np
import pytest

import oracle_lib as O
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,block", [(1, 1, 32), (33, 31, 32), (64, 32, 32), (31, 65, (16, 32)),
                                                (45, 7, (64, 3)), (5, 40, (1, 64)), (37, 29, (100, 100))])
def test_film_of_any_tiling(ctx, rtlib, width, height, block):
    s = scenes.cornell_box(width, height)
    g = rtlib.Scene(ctx, s)
    try:
        film = g.render(3, seed=5, block=block)
        batch = ctx.batch_render([(g, 3, dict(seed=5, block=block)), (g, 2, dict(seed=6))])
    finally:
        g.close()
    ref = O.OracleScene(s).render(3, seed=5, block=block)
    assert np.array_equal(film[..., 3], ref[..., 3])
    # as the film parity tests: rounding-level differences, a stated few flipped branches
    err = np.abs(film[..., :3] - ref[..., :3]) / np.maximum(np.abs(ref[..., :3]), 1e-3)
    assert np.mean(err.max(-1) > 1e-3) <= 0.02
    assert np.array_equal(batch[0], film)
