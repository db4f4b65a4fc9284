"""Closest-hit / any-hit parity of the CUDA traversal with the reference.

The golden fixtures hold the reference's own answers (BVH::intersect and
intersect_any run by oracle/ref_harness.cpp); larger batches are checked
against the oracle port, which test_oracle_pins.py pins to the reference
bit for bit.  The bar is bit-exact primitive ids and distances."""
import numpy as np
import pytest

from cpppt import scenes
from tests.golden.make_golden import SMALL_SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(SMALL_SCENES))
def test_closest_matches_reference_fixture(gpu_lib, golden, name):
    from cpppt.lib import GpuScene
    g = golden(f"{name}_ref.npz")
    sc = SMALL_SCENES[name]()
    gs = GpuScene(sc)
    idx, t, beta, gamma = gs.trace_closest(g["rays"])
    assert np.array_equal(idx, g["hit_index"]), np.nonzero(idx != g["hit_index"])[0][:10]
    assert np.array_equal(t.view(np.uint32), g["hit_t"].view(np.uint32))


@pytest.mark.parametrize("name", sorted(SMALL_SCENES))
def test_any_matches_reference_fixture(gpu_lib, golden, name):
    from cpppt.lib import GpuScene
    g = golden(f"{name}_ref.npz")
    gs = GpuScene(SMALL_SCENES[name]())
    occ = gs.trace_any(g["shadow_rays"])
    assert np.array_equal(occ, g["occluded"])


def test_closest_matches_oracle_large_batch(gpu_lib):
    from cpppt.lib import GpuScene
    from oracle.oracle import Oracle
    sc = scenes.soup(seed=2, n_spheres=400, freq=4, width=64, height=64)
    rays = scenes.hit_ray_batch(sc, 1 << 16, seed=11)
    oi, ot = Oracle("port").scene(sc).trace_closest(rays)
    gi, gt, _, _ = GpuScene(sc).trace_closest(rays)
    assert (oi >= 0).mean() > 0.9
    assert np.array_equal(gi, oi)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))


@pytest.mark.parametrize("config", ["cornell256", "soup1M"])
def test_full_size_ray_batch_matches_oracle(gpu_lib, config):
    """2^20 rays (seed 6: camera, secondary, edge/vertex and axis-parallel
    rays) on the Cornell box and on the 1M-triangle soup: closest-hit ids and
    distances bit-exact, any-hit answers identical for max_t around the hit."""
    from cpppt.lib import GpuScene
    from oracle.oracle import Oracle
    sc = scenes.cornell(256, 256) if config == "cornell256" else scenes.soup(seed=2)
    rays = scenes.hit_ray_batch(sc, 1 << 20, seed=6)
    osc = Oracle("port").scene(sc)
    oi, ot = osc.trace_closest(rays)
    gs = GpuScene(sc)
    gi, gt, _, _ = gs.trace_closest(rays)
    assert (oi >= 0).mean() > 0.5
    bad = np.nonzero(gi != oi)[0]
    assert bad.size == 0, (bad.size, bad[:8])
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))
    sh = rays.copy()
    rng = np.random.default_rng(7)
    hit = oi >= 0
    sh[hit, 6] = ot[hit] * rng.uniform(0.5, 1.5, size=hit.sum()).astype(np.float32)
    oo = osc.trace_any(sh)
    go = gs.trace_any(sh)
    assert 0.2 < oo.mean() < 0.9
    assert np.array_equal(go, oo)


def test_empty_and_degenerate_inputs(gpu_lib):
    from cpppt.lib import GpuScene
    sc = scenes.cornell(16, 16)
    gs = GpuScene(sc)
    idx, t, _, _ = gs.trace_closest(np.zeros((0, 7), np.float32))
    assert idx.size == 0
    # rays pointing away from everything and zero-length max_t
    rays = np.array([[0.5, 0.5, 5.0, 0, 0, 1, np.inf], [0.5, 0.5, 0.5, 0, 1, 0, 0.0]], np.float32)
    idx, t, _, _ = gs.trace_closest(rays)
    assert idx[0] == -1 and idx[1] == -1


@pytest.mark.parametrize("n", [1, 2, 31, 33, 151, 153, 1000, 4863, 4865, 9729, 77823, 77825, 155649])
def test_batch_sizes_around_the_ray_distribution(gpu_lib, n):
    """Batches around the warp, SM and fetch sizes of the traversal kernels:
    every ray is answered once, with the answer it has in any other batch."""
    from cpppt.lib import GpuScene
    from oracle.oracle import Oracle
    sc = scenes.soup(seed=2, n_spheres=60, freq=3, width=64, height=64)
    rays = scenes.hit_ray_batch(sc, n, seed=12)
    oi, ot = Oracle("port").scene(sc).trace_closest(rays)
    gs = GpuScene(sc)
    gi, gt, _, _ = gs.trace_closest(rays)
    assert np.array_equal(gi, oi)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))
    sh = rays.copy()
    sh[:, 6] = np.where(oi >= 0, ot * np.where(np.arange(n) % 2, 0.5, 1.5), 1.0).astype(np.float32)
    assert np.array_equal(gs.trace_any(sh), Oracle("port").scene(sc).trace_any(sh))


def test_stacks_beyond_their_shared_part(gpu_lib):
    """Overlapping spheres need more stack entries than the kernels keep in
    shared memory (13 of a closest-hit lane, 14 of an any-hit lane): with the
    stack limited to those the queries report an overflow, with the default
    limit they give the oracle's answers."""
    from cpppt.lib import GpuScene, PtError
    from oracle.oracle import Oracle
    sc = scenes.soup(seed=3, n_spheres=300, freq=4, width=64, height=64, extent=1.0)
    rays = scenes.hit_ray_batch(sc, 1 << 14, seed=13)
    osc = Oracle("port").scene(sc)
    oi, ot = osc.trace_closest(rays)
    sh = rays.copy()
    sh[:, 6] = np.where(oi >= 0, ot * np.where(np.arange(len(rays)) % 2, 0.99, 1.01), 1.0).astype(np.float32)
    gs = GpuScene(sc)
    for limit, query in ((13, lambda: gs.trace_closest(rays)), (14, lambda: gs.trace_any(sh))):
        assert gpu_lib.pt_debug_traversal_limits(gs.h, 0, limit) == 0
        with pytest.raises(PtError) as e:
            query()
        assert e.value.status == 4 and "stack overflow" in str(e.value)
    assert gpu_lib.pt_debug_traversal_limits(gs.h, 0, 0) == 0
    gi, gt, _, _ = gs.trace_closest(rays)
    assert np.array_equal(gi, oi)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))
    assert np.array_equal(gs.trace_any(sh), osc.trace_any(sh))


@pytest.mark.parametrize("n", [1, 33, 4863, 4864, 4865, 9728, 9729])
def test_device_batches_with_a_warp_per_ray(gpu_lib, n):
    """Batches of no more rays than the GPU has traversal warps (152 x 32) run
    without a cleared ray counter: the same answers as the host call, also
    after a batch that left the counter high, twice in a row."""
    torch = pytest.importorskip("torch")
    from cpppt.lib import GpuScene
    sc = scenes.soup(seed=2, n_spheres=100, freq=3, width=64, height=64)
    gs = GpuScene(sc)
    rays = scenes.hit_ray_batch(sc, 1 << 15, seed=11)
    d = torch.as_tensor(rays).cuda().contiguous()
    hits = torch.zeros(len(rays), 4, device="cuda")
    occ = torch.zeros(len(rays), dtype=torch.uint8, device="cuda")
    gs.trace_closest_device(d.data_ptr(), len(rays), hits.data_ptr())
    gs.trace_any_device(d.data_ptr(), len(rays), occ.data_ptr())
    torch.cuda.synchronize()  # a scene's batches share its counter: one stream at a time
    idx, t, _, _ = gs.trace_closest(rays[:n])
    blocked = gs.trace_any(rays[:n])
    gs.trace_closest_device(d.data_ptr(), len(rays), hits.data_ptr())
    for _ in range(2):
        hits.zero_()
        occ.zero_()
        torch.cuda.synchronize()
        gs.trace_closest_device(d.data_ptr(), n, hits.data_ptr())
        gs.trace_any_device(d.data_ptr(), n, occ.data_ptr())
        torch.cuda.synchronize()
        h = hits.cpu().numpy()
        assert np.array_equal(h[:n, 1].view(np.int32), idx)
        assert np.array_equal(h[:n, 0].view(np.uint32), t.view(np.uint32))
        assert np.array_equal(occ.cpu().numpy()[:n], blocked)
        assert (h[n:] == 0).all()
