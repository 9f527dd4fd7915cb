"""Per-kernel times of profiled renders: every ray that the statistics count is
traced in the kernels whose time and launches they report, however few the
paths."""
import numpy as np
import pytest

from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: scenes.cornell_box(32, 32), lambda: scenes.textured_room(41, 30)],
                         ids=["cornell", "textured"])
def test_profiled_times_cover_the_counted_rays(ctx, rtlib, make):
    g = rtlib.Scene(ctx, make())
    try:
        film = g.render(4, seed=2)
        plain = ctx.stats()
        ctx.set_profiling(1)
        timed = g.render(4, seed=2)
        st = ctx.stats()
        ctx.batch_render([(g, 4, dict(seed=2)), (g, 2, dict(seed=3))])
        batch = ctx.stats()
    finally:
        ctx.set_profiling(0)
        g.close()
    assert np.array_equal(timed, film)
    assert (st["closest_rays"], st["shadow_rays"]) == (plain["closest_rays"], plain["shadow_rays"])
    for s in (st, batch):
        # a launch of each kernel per round, and at least as many rounds as
        # bounces that the rays need
        assert s["trace_closest_launches"] >= 2 and s["trace_any_launches"] >= 2
        assert s["trace_closest_launches"] * s["paths"] >= s["closest_rays"]
        assert s["trace_closest_ms"] > 0 and s["trace_any_ms"] > 0 and s["shade_ms"] > 0
