"""Passes of one view against the oracle: scratch that overflows and the re-run, and rasters of many tiles."""
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

TWO_SIDED = np.stack([S.make_descriptor(tid=0, feature_flag=S.FLAG_TWO_SIDED)])


def oracle(sc):
    return O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0])


def check(got, ref):
    assert np.array_equal(got["depth"], ref["depth"]) and np.array_equal(got["id"], ref["id"])
    assert np.abs(got["rgba"].astype(int) - ref["rgba"].astype(int)).max() <= 1


@pytest.mark.parametrize("host", [False, True])
def test_overflow(host):
    """More bin entries than the first scratch holds: the counters reach the host, and the pass is run again whole."""
    rng = np.random.default_rng(7)
    w, h, n = 640, 480, 300
    x, y, z = rng.uniform(0, w - 250, n), rng.uniform(0, h - 250, n), rng.uniform(100, 3000, n)
    sc = tri_scene([screen_tri([a, a + 240, a], [b, b, b + 240], d, w, h) for a, b, d in zip(x, y, z)], w, h,
                   descs=TWO_SIDED)
    ref = oracle(sc)
    gs = GpuScene(sc)
    gs.set_tuning(S.PASS_VIEW, fine_max_tiles=256)
    for again in range(2):
        if host:
            pin = [torch.empty((h, w), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32) for _ in range(2)]
            rgba = torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True).numpy()
            check(gs.render_host(sc.cameras[0], sc.views[0], depth=pin[0], ids=pin[1], rgba=rgba), ref)
        else:
            check(gs.render(sc.cameras[0], sc.views[0]).numpy(), ref)
        st = gs.stats()
        assert st["retries"] >= 1 and st["view_records"] == n and st["view_bin_entries"] > 4 * (n + 1024)
        retries = st["retries"] if not again else retries
    assert gs.stats()["retries"] == retries  # the second frame fits
    gs.close()


@pytest.mark.parametrize("n_big,n_small,gap", [(3, 3000, 50.0), (40, 300, 0.01), (70, 0, 5.0)])
def test_many_tiles(n_big, n_small, gap):
    """More than 9,120 tiles (CTAs of 64 threads): tiles of one chunk and of several, and more covered pixels than a
    warp's list holds at once, many of them close behind one another."""
    rng = np.random.default_rng(n_big)
    w, h = 2001, 1239
    tl = []
    for i in rng.permutation(n_big):
        tl.append(screen_tri([-w, 3 * w, -w], [-h, -h, 3 * h], 500.0 + gap * i + rng.uniform(0, gap, 3), w, h))
    for _ in range(n_small):
        c, r, a = rng.uniform(0, 1, 2) * (w, h), rng.uniform(0.5, 30.0), rng.uniform(0, 2 * np.pi, 3)
        tl.append(screen_tri(c[0] + r * np.cos(a), c[1] + r * np.sin(a), rng.uniform(400, 500 + gap * n_big), w, h))
    sc = tri_scene(tl, w, h, descs=TWO_SIDED)
    ref = oracle(sc)
    gs = GpuScene(sc)
    check(gs.render(sc.cameras[0], sc.views[0]).numpy(), ref)
    gs.close()
