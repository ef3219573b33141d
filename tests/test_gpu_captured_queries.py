"""Ray queries captured into a CUDA graph on the caller's stream: the graph replayed after
xb_refit_mesh returns the refitted scene's hits. The refit rewrites the scene's arrays in place, so
a captured launch must read from them all that a refit changes: the moved mesh leaves its old
bounds, so the TLAS root's box, its leaves and the instances' order change."""
import numpy as np
import pytest

import xenon_b200 as xb
from xenon_b200 import HostScene, abi, scenes

pytestmark = pytest.mark.gpu


class _Query:
    """A query of fixed rays on a stream of its own, captured once."""

    def __init__(self, r, rays, mode, form):
        import torch
        self.torch, self.n = torch, len(rays)
        self.rays = torch.from_numpy(rays.view(np.uint8).reshape(-1).copy()).cuda()
        self.hits = torch.zeros(self.n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        self.stream = torch.cuda.Stream()
        call = xb.lib().xb_trace_rays_device if form == "device" else xb.lib().xb_trace_rays_noalloc

        def launch():
            xb.native.check(call(r.h, self.rays.data_ptr(), self.n, self.hits.data_ptr(), mode,
                                 self.stream.cuda_stream), r.h)
        torch.cuda.synchronize()
        launch()                     # outside a capture first, as xb_trace_rays_noalloc asks
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=self.stream):
            launch()

    def replay(self):
        self.hits.zero_()
        self.torch.cuda.synchronize()
        self.graph.replay()
        self.torch.cuda.synchronize()
        return self.hits.cpu().numpy().view(abi.HIT_DTYPE)


SCENES = {
    "icosphere": lambda: scenes.icosphere_scene(level=4),
    "grid": lambda: scenes.instanced_grid(grid=4, levels=(3, 3, 4, 4), with_prims=True),
}


@pytest.mark.parametrize("form", ["device", "noalloc"])
@pytest.mark.parametrize("mode", [abi.XB_TRACE_CLOSEST, abi.XB_TRACE_ANY])
@pytest.mark.parametrize("name", list(SCENES))
def test_captured_query_replays_after_a_refit(name, mode, form):
    desc = SCENES[name]()
    host = HostScene.from_desc(desc)
    used = {i[0] for i in desc.instances} or set(range(len(desc.meshes)))
    lit = {l[0] for l in desc.lights}
    mesh = max((len(m.positions), i) for i, m in enumerate(desc.meshes) if i in used - lit)[1]
    pos = abi.view_arrays(host.view())["meshes"][mesh]["pos"]
    lo, hi = scenes.scene_bounds(desc)
    up = np.float32(3.0) * (hi - lo)
    rays = np.concatenate([scenes.random_rays((lo, hi), 1 << 13, seed=5),
                           scenes.random_rays((lo + up, hi + up), 1 << 13, seed=6),
                           scenes.random_rays((lo, hi + up), 1 << 13, seed=7)])
    r = xb.Renderer(16, 16)
    r.upload_scene(host)
    q = _Query(r, rays, mode, form)
    assert q.replay().tobytes() == r.trace_rays(rays, mode).tobytes()
    for new in (pos + up, (0.2 * pos - 0.5 * up).astype(np.float32), pos):
        r.refit_mesh(mesh, new)
        host.refit_mesh(mesh, new)
        fresh = xb.Renderer(16, 16)
        fresh.upload_scene(host)
        want = fresh.trace_rays(rays, mode)
        assert r.trace_rays(rays, mode).tobytes() == want.tobytes()
        got = q.replay()
        assert np.array_equal(np.isfinite(got["t"]), np.isfinite(want["t"]))
        assert got.tobytes() == want.tobytes()
