"""What a scene counts against a server's memory budget: no more than the
figures that budgets have been planned by (40 bytes of vertex and mesh record per
triangle, 16 of colour and CDF per environment texel), so that a budget holds
the jobs that it held."""
import numpy as np
import pytest

import oracle_lib as O
import raytracer_gb300 as R
from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": (lambda: scenes.cornell_box(64, 48), False, 13592),
    "smooth": (lambda: scenes.cornell_smooth(64, 48), False, 15472),
    "textured": (lambda: scenes.textured_room(64, 48), False, 64652),
    "delta_lights": (lambda: scenes.cornell_delta_lights(64, 48), False, 14248),
    "volume": (lambda: scenes.volume_grid(64, 48, res=32), False, 141284),
    "planes": (lambda: scenes.plane_room(64, 48, textured=True), False, 20492),
    "icosphere": (lambda: scenes.displaced_icosphere(level=5, width=64, height=48, env_size=(256, 128)), False, 5793070),
    "icosphere_device_tree": (lambda: scenes.displaced_icosphere(level=5, width=64, height=48, env_size=(256, 128)), True,
                              3883982),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_scene_bytes(ctx, rtlib, name):
    make, device_tree, nbytes = SCENES[name]
    ctx.set_bvh_builder(device_tree)
    try:
        g = rtlib.Scene(ctx, make())
        got = g.info()["device_bytes"]
        g.close()
    finally:
        ctx.set_bvh_builder(False)
    assert got <= nbytes


def test_budget_admits_the_job_that_just_fits(ctx, rtlib):
    """A budget of the path state and one job's scene, at its planned figure,
    and film, to the byte, takes the job; a byte less than it counts refuses it."""
    make, _, nbytes = SCENES["icosphere"]
    g = rtlib.Scene(ctx, make())
    t = ctx.get_tuning()
    fixed = R.path_state_bytes(0) * t["wave_paths"] + R.path_state_bytes(1) * t["lane_wave_paths"]
    need = fixed + nbytes + 64 * 48 * 16
    srv = rtlib.Server(ctx, lanes=1, device_budget_bytes=need)
    info, film = srv.wait(srv.submit(g, 2, seed=1))
    srv.stop()
    assert info["state"] == rtlib.JOB_DONE and film is not None
    srv = rtlib.Server(ctx, lanes=1, device_budget_bytes=need - nbytes + g.info()["device_bytes"] - 1)
    with pytest.raises(rtlib.RtError) as e:
        srv.submit(g, 2, seed=1)
    assert e.value.status == 3
    srv.stop()
    g.close()


def _crowded(s, bsdfs):
    """s with 520 one-triangle meshes and 1030 point lights beside it, and
    diffuse BSDFs, unused, up to `bsdfs`."""
    for k in range(1030):
        s.add_point_light((0.2 + 0.0005 * k, 0.7, 0.4), (1e-3, 1e-3, 1e-3))
    wall = s.add_bsdf(D.bsdf(D.BSDF_DIFFUSE, albedo=(0.4, 0.5, 0.6)))
    for k in range(520):
        x, z = 0.1 + 0.03 * (k % 26), 0.1 + 0.03 * (k // 26)
        s.add_mesh(np.array([(x, 0.02, z), (x + 0.02, 0.03, z), (x, 0.04, z + 0.02)], np.float32),
                   np.array([(0, 1, 2)], np.int32), bsdf=wall)
    while len(s.bsdfs) < bsdfs:
        s.add_bsdf(D.bsdf(D.BSDF_DIFFUSE, albedo=(0.1, 0.1, 0.1)))
    return s


@pytest.mark.parametrize("make", [lambda: scenes.textured_room(40, 32), lambda: scenes.volume_grid(36, 28, res=16),
                                  lambda: scenes.cornell_smooth(40, 32)], ids=["textured", "volume", "smooth"])
def test_triangle_words_with_and_without_room(ctx, rtlib, make):
    """A triangle's BSDF, light and mesh in one word of its record (few BSDFs)
    and, where their numbers do not fit, looked up in its mesh (4096 BSDFs, 1030
    lights, 520 meshes take 34 bits): the same film."""
    films = []
    for bsdfs in (16, 4096):
        s = _crowded(make(), bsdfs)
        g = rtlib.Scene(ctx, s)
        films.append((g.render(3, seed=4), g.render(3, seed=4, max_depth=2)))
        g.close()
    assert np.array_equal(films[0][0], films[1][0]) and np.array_equal(films[0][1], films[1][1])
    ref = O.OracleScene(_crowded(make(), 16)).render(3, seed=4, max_depth=2)
    assert np.array_equal(films[0][1][..., 3], ref[..., 3])
    err = np.abs(films[0][1][..., :3] - ref[..., :3]) / np.maximum(np.abs(ref[..., :3]), 1e-3)
    assert np.mean(err.max(-1) > 1e-3) <= 0.03
