"""The traversal's own forms against the CPU restatement of the reference's loops, byte for byte:
rays that the packed slab test does not take (axis-parallel and denormal directions, signed zeros,
infinite and NaN components), origins on box planes, intervals that are empty or NaN; boxes that
hold NaNs or are inverted; leaves too large for a stack entry; records at 4-byte aligned
addresses; and batches around a warp's and a block's size."""
import ctypes

import numpy as np
import pytest

from oracle import port
from xenon_b200 import HostScene, Renderer, XenonError, abi, camera, raybatch, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda: scenes.cornell(),
    "prims": lambda: scenes.prim_showcase(),
    "icosphere": lambda: scenes.icosphere_scene(level=5),
    "grid": lambda: scenes.instanced_grid(grid=4, levels=(3, 3, 4, 4), with_prims=True),
}


def _rays(desc, n, seed):
    """Camera rays, incoherent rays and the special ones, shuffled so that warps mix them."""
    rng = np.random.default_rng(seed)
    cam = camera(desc.eye, desc.target, desc.fov, desc.width / desc.height)
    pts = np.concatenate([m.positions for m in desc.meshes] + [np.float32([[0, 1, 0], [1, 2, -1]])])
    lo, hi = pts.min(0), pts.max(0)
    k = n // 4
    a = raybatch.camera_rays(cam, desc.width, desc.height, k, seed)
    b = scenes.random_rays((lo, hi), k, seed + 1)
    # from vertices (on box planes), along the axes with zeros of either sign or denormals
    d = np.zeros((k, 3), np.float32)
    d[np.arange(k), rng.integers(0, 3, k)] = rng.choice([-1.0, 1.0], k)
    small = rng.choice(np.float32([0.0, -0.0, 1e-42, -1e-42, 1e-30]), (k, 3))
    d = np.where(d == 0, small, d).astype(np.float32)
    c = abi.make_rays(pts[rng.integers(0, len(pts), k)] + rng.choice(np.float32([0, 0, 1e-3]), (k, 3)), d)
    # one odd value per ray in a camera or an incoherent ray
    e = np.concatenate([a[: k // 2], b[: k // 2]]).copy()
    vals = np.float32([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e38, -1e38, 1e-40])
    for i in range(len(e)):
        f = ("org", "dir", "tmin", "tmax")[rng.integers(4)]
        x = vals[rng.integers(len(vals))]
        if f in ("org", "dir"):
            e[f][i, rng.integers(3)] = x
        else:
            e[f][i] = x if f == "tmax" else rng.choice(np.float32([np.inf, -np.inf, np.nan, 0.0, -3.0, 7.0]))
    rays = np.concatenate([a, b, c, e])
    rng.shuffle(rays)
    return rays


def _same(r, view, rays, count=True):
    r.upload_scene(view)
    ps = port.PortScene(view)
    r.reset_profile()
    got = r.trace_rays(rays, abi.XB_TRACE_CLOSEST)
    p = r.profile()
    want, work = ps.trace(rays, abi.XB_TRACE_CLOSEST)
    for f in ("prim_id", "instance_id"):
        assert np.array_equal(got[f], want[f]), (f, np.nonzero(got[f] != want[f])[0][:5])
    assert got["t"].tobytes() == want["t"].tobytes()
    if count:
        assert [p.ext_blas_nodes, p.ext_tris, p.ext_tlas_nodes, p.ext_instances] == [int(w) for w in work]
    any_got = r.trace_rays(rays, abi.XB_TRACE_ANY)
    any_want, _ = ps.trace(rays, abi.XB_TRACE_ANY)
    assert np.array_equal(np.isfinite(any_got["t"]), np.isfinite(any_want["t"]))
    return got


@pytest.mark.parametrize("flags", [0, abi.XB_FLAG_THREAD_PER_RAY])
@pytest.mark.parametrize("name", list(SCENES))
def test_odd_rays_match_the_oracle(name, flags):
    desc = SCENES[name]()
    r = Renderer(16, 16, flags=flags)
    got = _same(r, HostScene.from_desc(desc).view(), _rays(desc, 1 << 15, 3))
    assert (got["prim_id"] >= 0).mean() > 0.1


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 4097])
def test_batch_sizes_match_the_oracle(n):
    desc = SCENES["grid"]()
    rays = _rays(desc, 1 << 14, 5)[:n]
    _same(Renderer(16, 16), HostScene.from_desc(desc).view(), rays)


def _nodes(ptr, n):
    """The host scene's nodes, to be changed in place."""
    return np.frombuffer((ctypes.c_char * (n * 32)).from_address(ptr), abi.NODE_DTYPE)


@pytest.mark.parametrize("kind", ["blas_nan", "tlas_inverted", "blas_not_nested"])
def test_unusual_boxes_match_the_oracle(kind):
    desc = SCENES["grid"]()
    hs = HostScene.from_desc(desc)
    v = hs.view()
    rng = np.random.default_rng(8)
    if kind == "tlas_inverted":
        nd = _nodes(v.tlas_nodes, v.num_tlas_nodes)
        i = int(np.nonzero(nd["count"] > 0)[0][3])
        nd["mn"][i], nd["mx"][i] = np.inf, -np.inf
    else:
        for m in range(v.num_meshes):
            nd = _nodes(v.meshes[m].blas_nodes, v.meshes[m].num_blas_nodes)
            pick = rng.random(len(nd)) < 0.1
            if kind == "blas_nan":
                nd["mx"][pick, 1] = np.nan
            else:
                nd["mx"][pick] -= 0.3 * (nd["mx"][pick] - nd["mn"][pick])
    _same(Renderer(16, 16), v, _rays(desc, 1 << 14, 9))


@pytest.mark.parametrize("kind", ["blas", "tlas"])
def test_large_leaves_match_the_oracle(kind):
    """A BLAS leaf of 20 triangles and a TLAS leaf of 22 instances do not fit a stack entry."""
    desc = scenes.icosphere_scene(level=0) if kind == "blas" else SCENES["grid"]()
    hs = HostScene.from_desc(desc)
    v = hs.view()
    if kind == "blas":
        nd, n = _nodes(v.meshes[0].blas_nodes, v.meshes[0].num_blas_nodes), v.meshes[0].num_triangles
    else:
        nd, n = _nodes(v.tlas_nodes, v.num_tlas_nodes), v.num_instances
    assert n >= 15
    nd["child"][0], nd["count"][0] = 0, n
    r = Renderer(16, 16)
    rays = _rays(desc, 1 << 14, 11)
    want = _same(r, v, rays)
    if kind == "blas":      # the refit keeps the leaf
        r.refit_mesh(0, abi.view_arrays(v)["meshes"][0]["pos"])
        assert r.trace_rays(rays).tobytes() == want.tobytes()


def test_tlas_node_with_two_parents_is_refused():
    hs = HostScene.from_desc(SCENES["grid"]())
    v = hs.view()
    nd = _nodes(v.tlas_nodes, v.num_tlas_nodes)
    inner = np.nonzero(nd["count"] == 0)[0]
    nd["child"][inner[-1]] = nd["child"][inner[0]]
    r = Renderer(16, 16)
    with pytest.raises(XenonError) as e:
        r.upload_scene(v)
    assert e.value.code == abi.XB_E_INVALID


@pytest.mark.parametrize("mode", [abi.XB_TRACE_CLOSEST, abi.XB_TRACE_ANY])
def test_records_at_4_byte_alignment(mode):
    import torch
    desc = SCENES["grid"]()
    r = Renderer(16, 16)
    r.upload_scene(HostScene.from_desc(desc))
    rays = _rays(desc, 4000, 13)
    want = r.trace_rays(rays, mode)
    src = torch.zeros(rays.nbytes // 4 + 4, dtype=torch.int32, device="cuda")
    out = torch.zeros(len(rays) * 16 + 4, dtype=torch.int32, device="cuda")
    src[1:1 + rays.nbytes // 4] = torch.from_numpy(rays.view(np.int32).reshape(-1)).cuda()
    torch.cuda.synchronize()
    r.trace_rays_device(src.data_ptr() + 4, len(rays), out.data_ptr() + 4, mode)
    r.sync()
    assert out[1:1 + len(rays) * 16].cpu().numpy().tobytes() == want.tobytes()
    assert int(out[0]) == 0 and not out[1 + len(rays) * 16:].any()


def _below(nd, i):
    """The nodes that the walk from node i reaches."""
    seen, todo = set(), [int(i)]
    while todo:
        k = todo.pop()
        if k in seen:
            continue
        seen.add(k)
        if nd["count"][k] == 0:
            todo += [int(nd["child"][k]), int(nd["child"][k]) + 1]
    return seen


def _axis(nd, i):
    e = nd["mx"][i] - nd["mn"][i]
    return 0 if e[0] > e[1] and e[0] > e[2] else (1 if e[1] > e[2] else 2)


@pytest.mark.parametrize("kind", ["same_axis", "other_axis", "shifted", "many", "spare_nodes"])
def test_tlas_nodes_that_share_children_match_the_oracle(kind):
    """A TLAS whose nodes form no tree, but whose walk ends: a child pair with two parents (which
    order it along the same axis, or along different ones), two pairs with one node in common,
    many shared pairs, and nodes that no walk reaches."""
    desc = scenes.instanced_grid(grid=6, levels=(2, 2, 3, 3), with_prims=True)
    hs = HostScene.from_desc(desc)
    v = hs.view()
    n = v.num_tlas_nodes
    nd = np.concatenate([_nodes(v.tlas_nodes, n).copy(), np.zeros(5, abi.NODE_DTYPE)])
    nd["child"][n + 1:n + 3] = 1          # spare interior nodes, of which two share the root's children
    rng = np.random.default_rng(3)
    inner = np.nonzero(nd["count"][:n] == 0)[0]
    shared = 0
    if kind != "spare_nodes":
        pairs = [(a, b) for a in inner[1:] for b in inner[1:] if a != b]
        rng.shuffle(pairs)
        for a, b in pairs:
            c = int(nd["child"][b]) + (1 if kind == "shifted" else 0)
            if c + 1 >= n or a in _below(nd, c) or a in _below(nd, c + 1) or c == nd["child"][a]:
                continue
            if kind == "same_axis" and _axis(nd, a) != _axis(nd, b):
                continue
            if kind == "other_axis" and _axis(nd, a) == _axis(nd, b):
                continue
            nd["child"][a] = c
            shared += 1
            if shared == (8 if kind == "many" else 1):
                break
        assert shared > 0
    if kind == "spare_nodes":
        v.num_tlas_nodes = len(nd)
    v.tlas_nodes = nd.ctypes.data
    _same(Renderer(16, 16), v, _rays(desc, 1 << 14, 21))
