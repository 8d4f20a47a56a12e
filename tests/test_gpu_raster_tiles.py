"""Tiles the rasteriser treats specially: records that cover whole tiles and hide others, more
records than one chunk stages, more covered pixels than the id pass keeps, ragged edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from openclrenderer_gb300 import structs as S  # noqa: E402
from openclrenderer_gb300.pipeline import GpuScene  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.scene_util import screen_tri, tri_scene  # noqa: E402

TWO_SIDED = [S.make_descriptor(tid=0, feature_flag=S.FLAG_TWO_SIDED)]


def layers(w, h, n_big, n_small, gap, seed):
    """n_big tilted screen-covering triangles `gap` apart in depth (0: all coplanar), and small ones between them."""
    rng = np.random.default_rng(seed)
    tl = []
    for i in rng.permutation(n_big):
        z = 500.0 + gap * i + rng.uniform(0, 2.0, 3) * (gap > 0)
        tl.append(screen_tri([-w, 3 * w, -w], [-h, -h, 3 * h], z, w, h))
    for _ in range(n_small):
        c, r = rng.uniform(0, 1, 2) * (w, h), rng.uniform(0.5, 20.0)
        a = rng.uniform(0, 2 * np.pi, 3)
        tl.append(screen_tri(c[0] + r * np.cos(a), c[1] + r * np.sin(a), rng.uniform(400, 500 + gap * n_big + 100), w, h))
    return tri_scene(tl, w, h, descs=np.stack(TWO_SIDED))


@pytest.mark.parametrize("w,h", [(2, 2), (16, 16), (17, 33), (130, 47), (129, 64)])
@pytest.mark.parametrize("n_big,n_small,gap", [(1, 0, 1.0), (3, 40, 50.0), (150, 300, 5.0), (300, 0, 0.0), (600, 500, 0.01)])
def test_layers(w, h, n_big, n_small, gap):
    sc = layers(w, h, n_big, n_small, gap, seed=w + n_big)
    gs = GpuScene(sc)
    ref = O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0])
    for threads in (128, 256, 512):
        gs.set_tuning(S.PASS_VIEW, raster_threads=threads)
        got = gs.render(sc.cameras[0], sc.views[0]).numpy()
        assert np.array_equal(got["depth"], ref["depth"])
        assert np.array_equal(got["id"], ref["id"])
        assert np.abs(got["rgba"].astype(int) - ref["rgba"].astype(int)).max() <= 1
    gs.close()


def test_samples_count_hidden_records():
    """view_samples counts every covered (record, pixel) pair, hidden ones too: the sum over the records alone."""
    sc = layers(75, 50, 40, 60, 30.0, seed=9)
    gs = GpuScene(sc)
    gs.render(sc.cameras[0], sc.views[0])
    total, alone = gs.stats()["view_samples"], 0
    for t in range(len(sc.tris)):
        gs.set_triangles(sc.tris[t:t + 1])
        alone += int((gs.render(sc.cameras[0], sc.views[0]).numpy()["depth"] != 0xFFFFFFFF).sum())
    assert total == alone
    gs.close()


def test_hidden_cube_face_records():
    """Cubemap tiles with walls behind one another."""
    tl = []
    for z in (300.0, 420.0, 360.0, 300.5, 900.0):
        tl.append([(-2000, -2000, z), (6000, -2000, z), (-2000, 6000, z)])
        tl.append([(z, -2000, -2000), (z, 6000, -2000), (z, -2000, 6000)])
    sc = tri_scene(tl, 64, 48, descs=np.stack(TWO_SIDED),
                   lights=np.stack([S.make_light((0, 0, 0), radius=5000.0, shadow=1)]))
    gs = GpuScene(sc)
    gs.shadow_pass()
    dyn, _ = O.shadow(sc)
    assert np.array_equal(gs.cubemaps()[:len(dyn)], dyn)
    gs.close()


def test_triangles_without_a_pixel():
    """Triangles that round to a line or a point are counted as visible and draw nothing."""
    rng = np.random.default_rng(4)
    w, h = 200, 120
    tl = []
    for i in range(300):
        c = rng.integers(5, (w - 5, h - 5))
        r = rng.uniform(-0.4, 0.4, (2, 3))
        if i % 3 == 0:  # three points of one pixel row
            r[0] = (0, 3.0, 7.0)
        tl.append(screen_tri(c[0] + r[0], c[1] + r[1], rng.uniform(100, 900), w, h))
    sc = tri_scene(tl, w, h, descs=np.stack(TWO_SIDED))
    gs = GpuScene(sc)
    got = gs.render(sc.cameras[0], sc.views[0]).numpy()
    ref = O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0])
    assert (ref["depth"] == 0xFFFFFFFF).all() and np.array_equal(got["depth"], ref["depth"])
    st = gs.stats()
    assert st["view_records"] == 300 and st["view_samples"] == 0 and st["fragments_ref"] == ref["fragments"]
    gs.close()


@pytest.mark.parametrize("n", [900, 9000])
def test_coarse_records(n):
    """Every record in the coarse bins: listed at the end of the bins (900), or too many for that (9000)."""
    rng = np.random.default_rng(n)
    w, h, leg = 640, 480, 60
    x, y, z = rng.uniform(0, w - leg, n), rng.uniform(0, h - leg, n), rng.uniform(100, 3000, n)
    sc = tri_scene([screen_tri([a, a + leg, a], [b, b, b + leg], d, w, h) for a, b, d in zip(x, y, z)], w, h,
                   descs=np.stack(TWO_SIDED))
    gs = GpuScene(sc)
    gs.set_tuning(S.PASS_VIEW, fine_max_tiles=1, coarse_tile=64)
    got = gs.render(sc.cameras[0], sc.views[0]).numpy()
    ref = O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0])
    assert np.array_equal(got["depth"], ref["depth"]) and np.array_equal(got["id"], ref["id"])
    st, cap = gs.stats(), 4 * (n + 1024)
    assert st["retries"] == 0 and st["view_records"] == n and (st["view_bin_entries"] + n > cap) == (n == 9000)
    gs.close()


@pytest.mark.parametrize("sizes", [[(2001, 1239)], [(1500, 1100), (1201, 907)]])
@pytest.mark.parametrize("n_big,n_small,gap", [(1, 40, 1.0), (3, 4000, 50.0), (70, 300, 5.0), (140, 0, 0.0)])
def test_many_tiles(sizes, n_big, n_small, gap):
    """Passes of more than 9,120 tiles (CTAs of 64 threads) against those of 256: one view, and views of two sizes."""
    w, h = sizes[0]
    sc = layers(w, h, n_big, n_small, gap, seed=n_big)
    gs = GpuScene(sc)
    cams, views = [sc.cameras[0]] * len(sizes), [S.make_view(a, b, 90.0) for a, b in sizes]
    outs, samples = {}, {}
    for threads in (256, 128):
        gs.set_tuning(S.PASS_VIEW, raster_threads=threads)
        if len(sizes) == 1:
            outs[threads] = [gs.render(cams[0], views[0], normals=True).numpy()]
        else:
            outs[threads] = [o.numpy() for o in gs.render_batch(cams, views)]
        samples[threads] = gs.stats()["view_samples"]
    assert samples[128] == samples[256]
    for a, b in zip(outs[256], outs[128]):
        assert (a["depth"] != 0xFFFFFFFF).any()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    gs.close()


@pytest.mark.parametrize("n_lights", [1, 2])
def test_many_cube_face_tiles(n_lights):
    """Lights in a room whose walls cover every tile of every face: lists of 24,576 tiles and more, by halves of a block."""
    rng = np.random.default_rng(n_lights)
    tl, size, cells = [], 3000.0, 12  # (a triangle goes to the faces its vertices lie in, so walls of many)
    for axis in range(3):
        for side in (-size, size):
            for cell in range(cells * cells):
                for tri in ((0, 1, 2), (1, 3, 2)):
                    t = []
                    for k in tri:
                        v = np.full(3, side)
                        v[(axis + 1) % 3] = size * (2 * (cell % cells + (k & 1)) / cells - 1)
                        v[(axis + 2) % 3] = size * (2 * (cell // cells + (k >> 1)) / cells - 1)
                        t.append(tuple(v))
                    tl.append(t)
    for _ in range(60):
        c = rng.uniform(-size, size, 3)
        tl.append([tuple(c + rng.uniform(-400, 400, 3)) for _ in range(3)])
    sc = tri_scene(tl, 64, 48, descs=np.stack(TWO_SIDED),
                   lights=np.stack([S.make_light((40.0 * i, -30.0 * i, 25.0), radius=9000.0, shadow=1)
                                    for i in range(n_lights)]))
    gs = GpuScene(sc)
    gs.shadow_pass()
    dyn, _ = O.shadow(sc)
    assert (dyn != 0xFFFFFFFF).mean() > 0.9
    assert np.array_equal(gs.cubemaps()[:len(dyn)], dyn)
    gs.close()


@pytest.mark.parametrize("offset", [0, 4, 2])
def test_ids_into_pinned_memory(offset):
    """Host ids written by the raster itself (pinned, 4-byte aligned) or copied (2 bytes off): the same, and no others."""
    w, h = 333, 257
    sc = layers(w, h, 1, 200, 40.0, seed=3)
    sc.tris = sc.tris[1:]  # (some tiles stay empty)
    gs = GpuScene(sc)
    dev = gs.render(sc.cameras[0], sc.views[0]).numpy()
    raw = torch.empty(4 * w * h + 16, dtype=torch.uint8, pin_memory=True).numpy()
    raw[:] = 0xA5
    ids = raw[offset:offset + 4 * w * h].view(np.uint32)
    for _ in range(2):
        got = gs.render_host(sc.cameras[0], sc.views[0], ids=ids)
        assert np.array_equal(ids.reshape(h, w), dev["id"]) and np.array_equal(got["depth"], dev["depth"])
    assert (raw[:offset] == 0xA5).all() and (raw[offset + 4 * w * h:] == 0xA5).all()
    gs.close()
