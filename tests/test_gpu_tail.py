"""Few paths: the kernels that run a round's remaining paths to their end
(k_pt_tail, k_vw_tail) against the wavefront's rounds.  Profiling level 2
(traversal counters) renders without them, so the same call gives both films;
they are equal bit for bit, and so are the ray counts."""
import numpy as np
import pytest

import oracle_lib as O
from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu

PT, VW = 32768, 8192   # the paths of a round up to which the tail kernels take it


def _delta_all():
    s = scenes.cornell_delta_lights(61, 47)
    s.integrator = dict(s.integrator, strategy=D.STRATEGY_ALL_LIGHTS)
    return s


def _microfacet():
    s = scenes.cornell_smooth(48, 40)
    s.meshes[3]["bsdf"] = s.add_bsdf(D.bsdf(D.BSDF_MICROFACET, distribution=D.DIST_GGX, alpha=0.3, albedo=(0.5, 0.3, 0.2),
                                            eta_int=1.5))
    s.meshes[4]["bsdf"] = s.add_bsdf(D.bsdf(D.BSDF_LAYERED, alpha=0.1, alpha_base=0.2, eta=scenes.AU_ETA, k=scenes.AU_K))
    return s


CASES = {
    # one path; exactly the line; one tile row of samples above it (the last
    # rounds end in the tail kernel)
    "one_path": (lambda: scenes.cornell_box(1, 1), 1),
    "at_the_line": (lambda: scenes.cornell_smooth(64, 64), PT // 4096),
    "above_the_line": (lambda: scenes.textured_room(53, 37), PT // (53 * 37) + 1),
    "few_deep": (lambda: scenes.displaced_icosphere(level=3, width=37, height=29, env_size=(64, 32), max_depth=16), 3),
    "many_deep": (lambda: scenes.displaced_icosphere(level=3, width=160, height=96, env_size=(64, 32), max_depth=16), 9),
    "all_lights": (_delta_all, 5),
    "planes": (lambda: scenes.plane_room(64, 48, textured=True), 12),
    "mixed_queue": (_microfacet, 20),
    "depth_0": (lambda: _depth(0), 3),
    "depth_1": (lambda: _depth(1), 3),
    "volume_below": (lambda: scenes.volume_grid(33, 31, res=16), 8),
    "volume_at": (lambda: scenes.volume_grid(64, 32, res=16), VW // 2048),
    "volume_above": (lambda: scenes.volume_grid(64, 33, res=16), 9),
}


def _depth(n):
    s = scenes.cornell_box(24, 20)
    s.integrator = dict(s.integrator, max_depth=n)
    return s


def _both(ctx, call):
    out = []
    for level in (2, 0):
        ctx.set_profiling(level)
        try:
            r = call()
            out.append((r, ctx.stats()))
        finally:
            ctx.set_profiling(0)
    return out


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("graphs", [0, 1])
def test_tail_film_equals_rounds(ctx, rtlib, case, graphs):
    make, spp = CASES[case]
    g = rtlib.Scene(ctx, make())
    try:
        ctx.set_graphs(graphs)
        (ref, a), (got, b) = _both(ctx, lambda: g.render(spp, seed=7))
    finally:
        ctx.set_graphs(0)
        g.close()
    assert np.array_equal(got, ref)
    assert (a["closest_rays"], a["shadow_rays"], a["paths"]) == (b["closest_rays"], b["shadow_rays"], b["paths"])


@pytest.mark.parametrize("n", [1, 33, PT, PT + 1])
def test_tail_paths_equal_rounds(ctx, rtlib, n):
    g = rtlib.Scene(ctx, scenes.cornell_smooth(64, 64))
    rng = np.random.default_rng(n)
    px, sm = rng.integers(0, 64 * 64, n), rng.integers(0, 99, n)
    try:
        (ref, _), (got, _) = _both(ctx, lambda: g.render_paths(px, sm, seed=3))
    finally:
        g.close()
    assert np.array_equal(got, ref)


def test_tail_batch_equals_rounds(ctx, rtlib):
    gs = [rtlib.Scene(ctx, scenes.displaced_icosphere(level=2 + k % 2, width=24 + 9 * k, height=20, seed=k,
                                                      env_size=(64, 32), max_depth=12)) for k in range(4)]
    jobs = [(g, 2 + 3 * k, dict(seed=k)) for k, g in enumerate(gs)]
    try:
        (ref, _), (got, _) = _both(ctx, lambda: ctx.batch_render(jobs))
    finally:
        for g in gs:
            g.close()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


ROUNDS = {   # small films whose every path the tail kernels would take
    "smooth": (lambda: scenes.cornell_smooth(40, 33), 4, 0.03),
    "textured": (lambda: scenes.textured_room(41, 30), 4, 0.03),
    "icosphere": (lambda: scenes.displaced_icosphere(level=4, width=40, height=30, env_size=(64, 32), max_depth=8), 4, 0.03),
    "all_lights": (_delta_all, 3, 0.03),
    "volume": (lambda: scenes.volume_grid(32, 30, res=16), 4, 0.03),
}


@pytest.mark.parametrize("case", sorted(ROUNDS))
def test_rounds_match_oracle(ctx, rtlib, case):
    """The wavefront's own rounds on small films (profiling level 2: no tail
    kernels) against the oracle: weights bitwise, colours as the film parity
    tests have them (a few paths flip a branch on a last-ulp difference)."""
    make, spp, max_bad = ROUNDS[case]
    s = make()
    g = rtlib.Scene(ctx, s)
    ctx.set_profiling(2)
    try:
        film = g.render(spp, seed=19, block=16)
    finally:
        ctx.set_profiling(0)
        g.close()
    ref = O.OracleScene(s).render(spp, seed=19, block=16)
    assert np.array_equal(film[..., 3], ref[..., 3])
    err = np.abs(film[..., :3] - ref[..., :3]) / np.maximum(np.abs(ref[..., :3]), 1e-3)
    assert np.mean(err.max(-1) > 1e-3) <= max_bad


@pytest.mark.parametrize("make", [lambda: scenes.textured_room(48, 40), lambda: scenes.plane_room(48, 40, textured=True)],
                         ids=["textured_room", "plane_room"])
def test_textured_queues_equal_mixed(ctx, rtlib, make):
    """Textured BSDFs shaded from their type's queue give the film of the
    mixed queue's run-time dispatch (a sort threshold above every round)."""
    g = rtlib.Scene(ctx, make())
    before = ctx.get_tuning()
    ctx.set_profiling(2)
    try:
        film = g.render(5, seed=23)
        ctx.set_tuning(sort_threshold=1 << 30)
        mixed = g.render(5, seed=23)
    finally:
        ctx.set_tuning(**before)
        ctx.set_profiling(0)
        g.close()
    assert np.array_equal(film, mixed)
