"""SD-tree guided rendering (PPG, row a14) on the GPU against the reference's
own PPG renderer (src/renderer/ppg.h:149-215, run by the oracle harness).

Both learn their SD-tree online from their own paths, so the trees differ
sample by sample; the one-sample MIS estimator's mean does not depend on the
guide, so the images must agree statistically: per-tile z-test on replica
means.  The host tree update is pinned bit for bit in test_sdtree_host.py."""
import numpy as np
import pytest

from cpppt import scenes
from tests.test_gpu_render import check_z, tile_means, ztest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,res", [("cornell", (32, 32)), ("slitroom", (32, 16))])
def test_ppg_matches_reference_ppg(gpu_lib, name, res):
    from cpppt.lib import MODE_SDTREE, GpuScene
    from oracle import oracle as orc
    from tests.golden.make_golden import SMALL_SCENES
    if not orc.reference_available():
        pytest.fail("reference harness missing (build with __graft_entry__.build())")
    sc = SMALL_SCENES[name]().with_resolution(*res)
    R, tile, spp_axis = 8, 8, 8
    ref = orc.Oracle("reference").scene(sc)
    r_imgs = np.stack([ref.render_ppg(spp_axis, 100 * (r + 1))[0] for r in range(R)])
    gs = GpuScene(sc)
    g_imgs = np.stack([gs.render(spp_axis * spp_axis, max_depth=32, seed=50 + r, mode=MODE_SDTREE)
                       for r in range(R)])
    assert np.isfinite(g_imgs).all()
    check_z(ztest(tile_means(g_imgs, tile), tile_means(r_imgs, tile)), max_abs=6.0, frac3=0.05)


def test_ppg_learns_and_reports_stats(gpu_lib):
    from cpppt.lib import MODE_SDTREE, GpuScene
    gs = GpuScene(scenes.cornell(64, 64))
    img = gs.render(256, max_depth=16, seed=3, mode=MODE_SDTREE)
    st = gs.stats()
    # passes of 1, 2, ..., 128 spp: 255 spp worth of paths
    assert st["paths"] == 64 * 64 * 255
    assert img.mean() > 0.05 and np.isfinite(img).all()


@pytest.mark.parametrize("res,depth", [((1, 1), 32), ((17, 15), 2), ((16, 16), 3), ((33, 31), 40)],
                         ids=["one_pixel", "partial_block", "full_block", "long_paths"])
def test_ppg_splats_by_vertex(gpu_lib, res, depth):
    """The splats of a CTA's finished paths, one thread per vertex: the tree
    they train, and with it the image, is the same from run to run, and the
    image's mean is that of BSDF sampling to the same depth (6 standard errors
    over 16 seeds)."""
    from cpppt.lib import MODE_PT, MODE_SDTREE, GpuScene
    gs = GpuScene(scenes.cornell(*res))
    guided = [gs.render(64, max_depth=depth, seed=s, mode=MODE_SDTREE) for s in range(16)]
    again = [gs.render(64, max_depth=depth, seed=s, mode=MODE_SDTREE) for s in range(16)]
    assert all(np.array_equal(a, b) for a, b in zip(guided, again))
    plain = [gs.render(64, max_depth=depth, seed=s, mode=MODE_PT) for s in range(16)]
    g, p = (np.array([x.astype(np.float64).mean() for x in v]) for v in (guided, plain))
    se = np.sqrt(g.var(ddof=1) / len(g) + p.var(ddof=1) / len(p))
    assert abs(g.mean() - p.mean()) <= 6 * se


def test_ppg_gives_its_records_back(gpu_lib):
    """The vertex records of long paths (36 B x 2^19 paths x 150 vertices, 2.8
    GB) are freed when the render returns; a short render's are kept (at most
    256 MB) and give the image of a fresh scene."""
    torch = pytest.importorskip("torch")
    from cpppt.lib import MODE_SDTREE, GpuScene
    gs = GpuScene(scenes.cornell(256, 256))
    gs.render(16, max_depth=4, seed=1)  # the wavefront's own buffers, which stay
    gs.render(16, max_depth=2, seed=1, mode=MODE_SDTREE)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    gs.render(16, max_depth=150, rr_start=3, seed=1, mode=MODE_SDTREE)
    assert before - torch.cuda.mem_get_info()[0] <= 256 << 20
    again = gs.render(16, max_depth=2, seed=5, mode=MODE_SDTREE)
    assert before - torch.cuda.mem_get_info()[0] <= 256 << 20
    fresh = GpuScene(scenes.cornell(256, 256)).render(16, max_depth=2, seed=5, mode=MODE_SDTREE)
    assert np.array_equal(again.view(np.uint32), fresh.view(np.uint32))


def _finished_paths(seed, lengths):
    """Paths whose backward products are powers of two in [1/16, 16]: every sum
    of fewer than 2^16 of them is exact in any order."""
    rng = np.random.default_rng(seed)
    out = []
    for n in lengths:
        pos = np.where(rng.random((n, 1)) < 0.7, rng.normal([2, 2, 2], 0.6, (n, 3)), rng.uniform(0, 10, (n, 3)))
        d = rng.normal([0.3, -0.2, 0.8], 0.7, (n, 3))
        d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-9)
        prod = 2.0 ** rng.integers(-4, 5, (n, 3))
        factor = prod.copy()
        factor[:-1] /= prod[1:]
        out.append(np.hstack([pos, d, factor]).astype(np.float32))
    return out


@pytest.mark.parametrize("rounds", [[], [30000, 60000], [20000, 50000, 120000]], ids=["one_leaf", "split", "deep"])
@pytest.mark.parametrize("lengths", [[1], [0, 0, 3], [7] * 255, [5] * 256, [4] * 257, "mixed", "long"], ids=str)
def test_device_splats_equal_the_hosts(gpu_lib, rounds, lengths):
    """Counts, flux and quadtree values of the device's splats of finished
    paths against the host tree's, exactly: partial blocks, paths without
    vertices, paths whose last vertex carries nothing, several spatial leaves
    in a warp."""
    from cpppt import lib
    from tests.test_sdtree_host import make_rounds
    rng = np.random.default_rng(4)
    if lengths == "mixed":
        lengths = rng.integers(0, 12, 3001)
    elif lengths == "long":
        lengths = [2000, 1, 1023, 0, 4097, 4]
    paths = _finished_paths(5, lengths)
    for p in paths[::5][1:]:
        p[-1:, 6:] = 0
    args = ([0, 0, 0], [10, 10, 10], make_rounds(7, rounds), paths)
    host, dev = (lib.sdtree_splat(*args, on_device=k) for k in (False, True))
    assert host["counts"].sum() == sum(len(p) for p in paths if len(p) and p[-1, 6:].max() > 0)
    assert len(rounds) == 0 or len(host["counts"]) > 1
    assert np.array_equal(dev["counts"], host["counts"])
    for key in ("values", "flux"):
        assert np.array_equal(dev[key].view(np.uint32), host[key].view(np.uint32)), key


def test_splats_of_long_paths_take_linear_time(gpu_lib):
    """64 paths of 8000 vertices against 64 of 2000: four times the work."""
    import time

    from cpppt import lib

    def ms(n):
        paths, best = _finished_paths(6, [n] * 64), 1e9
        for _ in range(4):
            t = time.perf_counter()
            lib.sdtree_splat([0, 0, 0], [10, 10, 10], [], paths, on_device=True)
            best = min(best, 1e3 * (time.perf_counter() - t))
        return best
    short, long = ms(2000), ms(8000)
    print(f"{short:.1f} ms, {long:.1f} ms")
    assert long <= 6 * short, (short, long)
