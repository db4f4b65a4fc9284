"""Device build of the reference-topology BVH (csrc/gpu_bvh.cu): the same
tree as BVH::build (bvh.h:151-216) -- leaf order (the tie-break ranks),
internal-node boxes in pre-order and each triangle's innermost internal
node -- bit for bit against the reference's own trees (golden fixtures), the
host build and the oracle, including -0.0 / +0.0 coordinates (the
reference's min / max keep the later of equal values) and a block of
coincident triangles (the reference's endless recursion becomes one leaf).
pt_scene_create builds every scene's tree this way, so the hit and image
tests run on it too."""
import numpy as np
import pytest

from cpppt import scenes
from tests.golden.make_golden import SMALL_SCENES

pytestmark = pytest.mark.gpu


def _same(a, b):
    order, boxes, pparent = a[:3]
    o_order, o_boxes, o_pparent = b[:3]
    assert np.array_equal(order, o_order)
    assert boxes.shape == o_boxes.shape
    assert np.array_equal(boxes.view(np.uint32), o_boxes.view(np.uint32))
    assert np.array_equal(pparent, o_pparent)


@pytest.mark.parametrize("name", sorted(SMALL_SCENES))
def test_device_build_matches_reference_fixture(gpu_lib, golden, name):
    from cpppt import lib
    g = golden(f"{name}_ref.npz")
    order, boxes, pparent, _ = lib.ref_topology_device(SMALL_SCENES[name]())
    _same((order, boxes, pparent), (g["leaf_order"], g["node_boxes"], g["prim_parent"]))


def test_device_build_matches_host_with_coincident_block(gpu_lib):
    from cpppt import lib
    sc = scenes.soup(seed=9, n_spheres=1000, freq=4, width=8, height=8)
    sc.triangles[1000:41000] = sc.triangles[7]  # 40000 coincident copies of one triangle
    dev = lib.ref_topology_device(sc)
    assert dev[3] > 10
    _same(dev, lib.ref_topology(sc))


def test_device_build_signed_zeros(gpu_lib):
    """Coordinates of 0.0 written as +0.0 and -0.0 in an irregular pattern:
    every min / max must keep the later of two equal values."""
    from cpppt import lib
    from oracle.oracle import Oracle
    sc = scenes.soup(seed=11, n_spheres=150, freq=3, width=8, height=8, extent=4.0)
    rng = np.random.default_rng(3)
    v = sc.vertices.copy()
    pick = rng.random(v.shape) < 0.25
    v[pick] = np.round(v[pick])  # many exact integers, among them zeros
    v[(v == 0) & (rng.random(v.shape) < 0.5)] = np.float32(-0.0)
    assert (np.signbit(v) & (v == 0)).sum() > 50
    sc.vertices = v
    dev = lib.ref_topology_device(sc)
    _same(dev, lib.ref_topology(sc))
    o_order, o_boxes, _, o_pparent = Oracle("port").scene(sc).bvh_dump()
    _same(dev, (o_order, o_boxes, o_pparent))


@pytest.mark.parametrize("make", [lambda: scenes.soup(seed=2),
                                  lambda: scenes.slit_room(seed=4, n_boxes=1000, box_subdiv=4)],
                         ids=["soup1M", "slitroom192k"])
def test_device_build_full_size(gpu_lib, make):
    from cpppt import lib
    sc = make()
    _same(lib.ref_topology_device(sc), lib.ref_topology(sc))


@pytest.mark.parametrize("n", [1, 3, 4, 7, 31, 32, 33, 34, 65, 129, 2047, 2048, 2049])
def test_device_build_at_node_size_limits(gpu_lib, n):
    """A leaf, a warp's node (up to 32), a CTA's (up to 2048), several CTAs'."""
    from dataclasses import replace

    from cpppt import lib
    sc = scenes.soup(seed=3, n_spheres=40, freq=3, width=8, height=8)
    tris = np.random.default_rng(n).permutation(sc.triangles)[:n]
    sc = replace(sc, triangles=np.ascontiguousarray(tris))  # geometry only: the tree builds read nothing else
    _same(lib.ref_topology_device(sc), lib.ref_topology(sc))


def _same_wide(sc):
    from cpppt import lib
    dn, do, dd, df = lib.wide_bvh(sc, on_device=True)
    hn, ho, hd, hf = lib.wide_bvh(sc, on_device=False)
    assert dn.shape == hn.shape, (dn.shape, hn.shape)
    assert np.array_equal(dn, hn)
    assert np.array_equal(do, ho)
    assert (dd, df) == (hd, hf)
    return dn


def _tiny(n, seed=0):
    sc = scenes.soup(seed=seed, n_spheres=4, freq=1, width=8, height=8)
    sc.triangles = sc.triangles[:n].copy()  # geometry only: the tree builds read nothing else
    return sc


@pytest.mark.parametrize("name", sorted(SMALL_SCENES))
def test_device_wide_tree_matches_host_small(gpu_lib, name):
    """Device binned-SAH build and 4-wide collapse (csrc/gpu_sah.cu): the
    host build's nodes, leaf order, depth and inflation, byte for byte."""
    _same_wide(SMALL_SCENES[name]())


@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 300])
def test_device_wide_tree_matches_host_tiny(gpu_lib, n):
    _same_wide(_tiny(n))


def test_device_wide_tree_coincident_and_flat(gpu_lib):
    """Blocks of coincident triangles (no SAH split: halved in insertion
    order, in the level-synchronous top levels for 40000 copies and inside a
    subtree for 100), a flat scene (one axis without extent) and signed
    zeros."""
    sc = scenes.soup(seed=9, n_spheres=1000, freq=4, width=8, height=8)
    sc.triangles[1000:41000] = sc.triangles[7]
    sc.triangles[50000:50100] = sc.triangles[9]
    _same_wide(sc)
    flat = scenes.soup(seed=12, n_spheres=200, freq=2, width=8, height=8)
    flat.vertices = flat.vertices.copy()
    flat.vertices[:, 2] = np.float32(3.0)
    _same_wide(flat)
    z = scenes.soup(seed=11, n_spheres=150, freq=3, width=8, height=8, extent=4.0)
    rng = np.random.default_rng(3)
    v = z.vertices.copy()
    pick = rng.random(v.shape) < 0.25
    v[pick] = np.round(v[pick])
    v[(v == 0) & (rng.random(v.shape) < 0.5)] = np.float32(-0.0)
    z.vertices = v
    _same_wide(z)


@pytest.mark.parametrize("make", [lambda: scenes.soup(seed=2),
                                  lambda: scenes.slit_room(seed=4, n_boxes=1000, box_subdiv=4)],
                         ids=["soup1M", "slitroom192k"])
def test_device_wide_tree_full_size(gpu_lib, make):
    """Full size, and the device build repeated: atomics decide only node
    numbering inside the build, never the output."""
    from cpppt import lib
    sc = make()
    nodes = _same_wide(sc)
    assert len(nodes) > 10000
    for _ in range(4):
        again = lib.wide_bvh(sc, on_device=True)[0]
        assert np.array_equal(again, nodes)


def _chain(links, per):
    """Clusters of `per` triangles along x, each three times closer to the origin."""
    from dataclasses import replace
    x = (np.float32(3) ** -np.arange(links, dtype=np.float32))[:, None] * (
        1 + np.float32(0.01) * np.arange(per, dtype=np.float32))
    x = x.reshape(-1)
    z = np.zeros_like(x)
    v = np.stack([np.stack([x, z, z], 1), np.stack([x, x * np.float32(.1), z], 1),
                  np.stack([x, z, x * np.float32(.1)], 1)], 1).reshape(-1, 3).astype(np.float32)
    n = len(v) // 3
    sc = scenes.soup(seed=5, n_spheres=2, freq=1, width=8, height=8)
    up, side = np.float32([[0, 0, 1]]), np.float32([[1, 0, 0]])
    return replace(sc, vertices=v, normals=np.repeat(up, len(v), 0), tangents=np.repeat(side, len(v), 0),
                   triangles=np.arange(len(v), dtype=np.int32).reshape(-1, 3),
                   mesh_tri_offset=np.array([0, n], np.int32), mesh_vert_offset=np.array([0, len(v)], np.int32),
                   mesh_material=np.array([0], np.int32))


@pytest.mark.parametrize("links,per,depth", [(15, 4000, 18), (19, 4000, 19), (24, 4000, 24)],
                         ids=["cheapest", "cheapest_too_deep", "both_too_deep"])
def test_wide_tree_at_depth_limit(gpu_lib, links, per, depth):
    """The cheapest collapse, or the largest-first one where the cheapest
    exceeds the traversal's depth (20; 21 levels for 19 links); a scene whose
    largest-first tree exceeds it is refused, though its cheapest would fit."""
    from cpppt import lib
    from oracle.oracle import Oracle
    sc = _chain(links, per)
    _same_wide(sc)
    assert lib.wide_bvh(sc, on_device=False)[2] == depth
    if depth > 20:
        with pytest.raises(lib.PtError, match="too deep"):
            lib.GpuScene(sc)
        return
    rays = scenes.hit_ray_batch(sc, 2048, seed=1)
    gi, gt, _, _ = lib.GpuScene(sc).trace_closest(rays)
    oi, ot = Oracle("port").scene(sc).trace_closest(rays)
    assert (oi >= 0).any()
    assert np.array_equal(gi, oi)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))


@pytest.mark.parametrize("n", [0, 1, 4, 5, 32, 33, 255, 256, 257, 3001])
def test_scene_arrays_at_block_edges(gpu_lib, n):
    """The scene's arrays, assembled on the device: hits of the first n
    triangles of a soup equal the oracle's bit for bit, and light areas and
    materials follow (a render of the same triangles is finite and, without
    triangles, black)."""
    from dataclasses import replace

    from cpppt.lib import GpuScene
    from oracle.oracle import Oracle
    full = scenes.soup(seed=5, n_spheres=60, freq=3, width=24, height=16)
    tris = np.random.default_rng(1).permutation(full.triangles)[:n]
    half = n // 2
    sc = replace(full, triangles=np.ascontiguousarray(tris), mesh_tri_offset=np.array([0, half, n], np.int32),
                 mesh_material=np.array([0, len(full.mat_kind) - 1], np.int32),
                 mesh_vert_offset=np.array([0, 0, len(full.vertices)], np.int32))
    rays = scenes.hit_ray_batch(full, 4096, seed=3)
    gs = GpuScene(sc)
    gi, gt, _, _ = gs.trace_closest(rays)
    img = gs.render(2, 4)
    assert np.isfinite(img).all()
    if n == 0:
        assert (gi < 0).all() and (img == 0).all()
        return
    oi, ot = Oracle("port").scene(sc).trace_closest(rays)
    assert np.array_equal(gi, oi)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))


def test_scene_without_tangents_uses_perpendicular(gpu_lib, monkeypatch):
    """A description without tangents renders as one with the unit vector
    perpendicular to each normal, computed here in 32 bits operation by
    operation: the same image bit for bit."""
    from dataclasses import replace

    from cpppt import lib
    sc = scenes.slit_room(n_boxes=12, width=48, height=32)
    f = np.float32
    n = sc.normals.astype(f)
    x = np.abs(n[:, 1]) < f(0.9)
    a = np.stack([np.where(x, 0, 1), np.where(x, 1, 0), np.zeros(len(n))], 1).astype(f)
    t = np.stack([a[:, 1] * n[:, 2] - a[:, 2] * n[:, 1], a[:, 2] * n[:, 0] - a[:, 0] * n[:, 2],
                  a[:, 0] * n[:, 1] - a[:, 1] * n[:, 0]], 1)
    inv = f(1) / np.sqrt((t[:, 0] * t[:, 0] + t[:, 1] * t[:, 1]) + t[:, 2] * t[:, 2])
    given = lib.GpuScene(replace(sc, tangents=t * inv[:, None])).render(8, 6)

    class NoTangents(lib.PtSceneDesc):
        def __setattr__(self, name, value):
            super().__setattr__(name, None if name == "tangents" else value)

    monkeypatch.setattr(lib, "PtSceneDesc", NoTangents)
    none = lib.GpuScene(sc).render(8, 6)
    assert given.max() > 0
    assert np.array_equal(given.view(np.uint32), none.view(np.uint32))
