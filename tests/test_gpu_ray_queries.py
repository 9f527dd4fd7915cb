"""Any-hit queries of rt_trace beside closest-hit ones, under every tree width:
counts around a warp and a block, ranges that stop before or start behind the
hit, on state that a render and the other kind of query have just used."""
import numpy as np
import pytest

import oracle_lib as O
from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(n, 3))
    o *= rng.uniform(1.5, 5.0, (n, 1)) / np.linalg.norm(o, axis=1, keepdims=True)
    o[:, 1] = np.abs(o[:, 1]) + 0.05
    d = rng.normal(size=(n, 3)) * 0.6 + np.array([0.0, 1.0, 0.0]) - o
    r = np.zeros(n, D.RAY_DTYPE)
    r["o"], r["d"], r["mint"], r["maxt"] = o, d / np.linalg.norm(d, axis=1, keepdims=True), 1e-4, 1e4
    return r


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 5000, 40001])
def test_anyhit_agrees_with_closest(ctx, rtlib, width, n):
    s = scenes.displaced_icosphere(level=4, width=40, height=30, env_size=(64, 32))
    g, o = rtlib.Scene(ctx, s), O.OracleScene(s)
    rays = _rays(n, n)
    try:
        ctx.set_bvh_width(width)
        film = g.render(2, seed=1)
        closest = g.trace(rays)
        hit = closest["prim"] != -1
        # all of them; ending just before the hit; starting just behind it
        assert np.array_equal(g.trace(rays, anyhit=True)["prim"] != -1, hit)
        before = rays.copy()
        before["maxt"] = np.where(hit, closest["t"] * np.float32(0.999), rays["maxt"])
        behind = rays.copy()
        behind["mint"] = np.where(hit, closest["t"] * np.float32(1.001), rays["mint"])
        for r in (before, behind):
            a = g.trace(r, anyhit=True)
            assert np.array_equal(a["prim"] != -1, g.trace(r)["prim"] != -1)
            assert np.array_equal(a["prim"] != -1, o.trace(r, anyhit=True)["prim"] != -1)
            assert not a["t"].any() and not a["u"].any() and not a["v"].any()
        assert not (g.trace(before, anyhit=True)["prim"] != -1)[hit].any()
        assert np.array_equal(g.trace(rays), closest)
        assert np.array_equal(g.render(2, seed=1), film)
    finally:
        ctx.set_bvh_width(2)
        g.close()
