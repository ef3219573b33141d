"""Renders after xb_refit_mesh on a renderer that keeps its captured bounce loops (tuning graph =
1): bit for bit the images of a fresh renderer with the refitted scene uploaded, for moves that
change the scene's bounds and moves that leave them, plain, guided (a fixed network) and views."""
import numpy as np
import pytest

import xenon_b200 as xb
from xenon_b200 import HostScene, abi, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "icosphere": lambda: scenes.icosphere_scene(level=4, width=96, height=54),
    "grid": lambda: scenes.instanced_grid(grid=3, levels=(3, 3, 4, 4), with_prims=True),
    "room": lambda: scenes.guiding_room(level=3, width=96, height=54),
}


def _renderer(host, guided):
    r = xb.Renderer(96, 54, max_bounces=6, min_bounces=3)
    r.set_tuning(graph=1)
    r.upload_scene(host)
    if guided:
        r.set_guiding(True, train_spp=-1, seed=4)
    return r


def _image(r, cam, form):
    if form == "views":
        return np.concatenate([i.reshape(-1) for i in r.render_views([(cam, 96, 54, 2), (cam, 33, 17, 3)])])
    r.reset()
    r.render_frame(cam, 2)
    return r.resolve().copy()


@pytest.mark.parametrize("form", ["plain", "guided", "views", "guided_views"])
@pytest.mark.parametrize("name", list(SCENES))
def test_render_after_refit_equals_a_fresh_upload(name, form):
    desc = SCENES[name]()
    cam = xb.camera(desc.eye, desc.target, desc.fov, 96 / 54)
    host = HostScene.from_desc(desc)
    used = {i[0] for i in desc.instances} or set(range(len(desc.meshes)))
    lit = {l[0] for l in desc.lights}
    mesh = max((len(m.positions), i) for i, m in enumerate(desc.meshes) if i in used - lit)[1]
    pos = abi.view_arrays(host.view())["meshes"][mesh]["pos"]
    centre = pos.mean(0)
    guided = form.startswith("guided")
    r = _renderer(host, guided)
    f = "views" if form.endswith("views") else "frame"
    first = _image(r, cam, f)
    assert np.array_equal(_image(r, cam, f), first)      # the kept loops replay
    changed = False
    for new in (centre + np.float32(0.8) * (pos - centre), centre + np.float32(6.0) * (pos - centre) + np.float32([0, 3, 0]),
                pos):
        new = new.astype(np.float32)
        r.refit_mesh(mesh, new)
        host.refit_mesh(mesh, new)
        got = _image(r, cam, f)
        fresh = _renderer(host, guided)
        want = _image(fresh, cam, f)
        fresh.close()
        assert np.array_equal(got, want)
        changed = changed or not np.array_equal(got, first)
    assert changed
    assert np.array_equal(got, first)
