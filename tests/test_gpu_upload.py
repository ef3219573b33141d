"""Scene upload: the device packs each mesh's arrays (small meshes go up as one copy, large ones
array by array). Traces through the packed scene equal the CPU restatement's over the caller's
arrays, and indices out of range are refused, after which a sound scene uploads."""
import ctypes

import numpy as np
import pytest

from oracle import port
from xenon_b200 import HostScene, Renderer, XenonError, abi, scenes

pytestmark = pytest.mark.gpu


def _array(ptr, n, dtype):
    """One of the host scene's arrays, to be changed in place."""
    return np.frombuffer((ctypes.c_char * (n * np.dtype(dtype).itemsize)).from_address(ctypes.cast(ptr, ctypes.c_void_p).value), dtype)


@pytest.mark.parametrize("level", [0, 3, 5, 6])   # 22 to 81,922 triangles: both sides of one copy
def test_packed_scene_traces_as_the_oracle(level):
    desc = scenes.icosphere_scene(level=level)
    extra = scenes.cornell()                      # more meshes, of other sizes, with normals and lights
    m0 = len(desc.materials)
    for name, m in zip(extra.material_names, extra.materials):
        desc.add_material(name, m)
    for mesh in extra.meshes:
        desc.add_mesh(scenes.MeshDesc(mesh.positions, mesh.indices, mesh.normals, None, m0 + mesh.default_mat))
    v = HostScene.from_desc(desc).view()
    rays = scenes.random_rays(scenes.scene_bounds(desc), 1 << 14, seed=level)
    r = Renderer(16, 16)
    r.upload_scene(v)
    got = r.trace_rays(rays)
    want, _ = port.PortScene(v).trace(rays, abi.XB_TRACE_CLOSEST)
    for f in ("prim_id", "instance_id", "mat_id", "front_face"):
        assert np.array_equal(got[f], want[f]), f
    for f in ("t", "u", "v", "normal", "geo_normal"):
        assert got[f].tobytes() == want[f].tobytes(), f


@pytest.mark.parametrize("level", [2, 6])
@pytest.mark.parametrize("what", ["leaf", "child", "prim", "vertex", "material"])
def test_bad_indices_are_refused(what, level):
    desc = scenes.icosphere_scene(level=level)
    v = HostScene.from_desc(desc).view()
    mv = v.meshes[0]
    nodes = _array(mv.blas_nodes, mv.num_blas_nodes, abi.NODE_DTYPE)
    if what == "leaf":
        nodes["child"][np.nonzero(nodes["count"] > 0)[0][-1]] = mv.num_triangles
    elif what == "child":
        nodes["child"][np.nonzero(nodes["count"] == 0)[0][-1]] = mv.num_blas_nodes
    elif what == "prim":
        _array(mv.blas_prims, mv.num_triangles, np.uint32)[-1] = mv.num_triangles
    elif what == "vertex":
        _array(mv.indices, 3 * mv.num_triangles, np.int32)[-1] = mv.num_vertices
    else:
        _array(mv.mat_ids, mv.num_triangles, np.int32)[-1] = v.num_materials
    r = Renderer(16, 16)
    with pytest.raises(XenonError) as e:
        r.upload_scene(v)
    assert e.value.code == abi.XB_E_INVALID
    r.upload_scene(HostScene.from_desc(desc))
    rays = scenes.random_rays(scenes.scene_bounds(desc), 256, seed=1)
    assert (r.trace_rays(rays)["prim_id"] >= 0).any()


@pytest.mark.parametrize("level", [2, 6])
@pytest.mark.parametrize("missing", ["ny", "nz"])
def test_a_missing_normal_component_is_zero(missing, level):
    """Normals of which one component's array is NULL: that component is 0, whatever device memory
    held before (a scene with all three was uploaded by the same renderer)."""
    desc = scenes.icosphere_scene(level=level)
    desc.meshes[0].normals = desc.meshes[0].positions / np.linalg.norm(desc.meshes[0].positions, axis=1, keepdims=True)
    rays = scenes.random_rays(scenes.scene_bounds(desc), 1 << 12, seed=3)
    hs = HostScene.from_desc(desc)
    v = hs.view()
    r = Renderer(16, 16)
    r.upload_scene(v)
    zeros = np.zeros(v.meshes[0].num_vertices, np.float32)
    setattr(v.meshes[0], missing, zeros.ctypes.data_as(ctypes.POINTER(ctypes.c_float)))
    want, _ = port.PortScene(v).trace(rays, abi.XB_TRACE_CLOSEST)
    setattr(v.meshes[0], missing, ctypes.POINTER(ctypes.c_float)())
    r.upload_scene(v)
    got = r.trace_rays(rays)
    assert (got["prim_id"] >= 0).mean() > 0.1
    assert got["normal"].tobytes() == want["normal"].tobytes()


def test_instances_without_a_tlas_hit_nothing_until_a_refit_builds_one():
    desc = scenes.instanced_grid(grid=3, levels=(3, 3, 3, 3), with_prims=True)
    rays = scenes.random_rays(scenes.scene_bounds(desc), 1 << 12, seed=4)
    hs = HostScene.from_desc(desc)
    v = hs.view()
    r = Renderer(16, 16)
    r.upload_scene(v)
    want = r.trace_rays(rays)
    assert (want["prim_id"] >= 0).mean() > 0.1
    lit = {l[0] for l in desc.lights}
    mesh = next(m for m in range(len(desc.meshes)) if m not in lit)
    pos = abi.view_arrays(v)["meshes"][mesh]["pos"]
    v.num_tlas_nodes = 0
    r.upload_scene(v)
    assert (r.trace_rays(rays)["prim_id"] < 0).all()
    r.refit_mesh(mesh, pos)
    assert r.trace_rays(rays).tobytes() == want.tobytes()
