"""Rows narrowed to spans for triangles whose vertices lie off the surface, against the oracle."""
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


def triangles(n, w, h, far, thin, seed):
    """Screen-space triangles along random lines through the view, up to `far` pixels long and `thin` wide."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        c, a = rng.uniform(0, 1, 2) * (w, h), rng.uniform(0, 2 * np.pi)
        d, q = rng.uniform(-far, far, 3), rng.uniform(-thin, thin, 3)
        out.append((c[0] + d * np.cos(a) - q * np.sin(a), c[1] + d * np.sin(a) + q * np.cos(a), rng.uniform(50, 3000)))
    return out


@pytest.mark.parametrize("w,h", [(17, 9), (333, 217), (1920, 1080)])
@pytest.mark.parametrize("far,thin", [(30.0, 30.0), (3000.0, 3.0), (3000.0, 3000.0), (200000.0, 60.0), (2000000.0, 1000.0)])
def test_views(w, h, far, thin):
    """Vertices on the surface, near it, and farther off than spans are taken for."""
    sc = tri_scene([screen_tri(x, y, z, w, h) for x, y, z in triangles(300, w, h, far, thin, seed=w)], w, h,
                   descs=TWO_SIDED)
    ref = O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0], shade=False)
    gs = GpuScene(sc)
    got = gs.render(sc.cameras[0], sc.views[0]).numpy()
    gs.close()
    assert (ref["depth"] != 0xFFFFFFFF).any()
    assert np.array_equal(got["depth"], ref["depth"]) and np.array_equal(got["id"], ref["id"])


@pytest.mark.parametrize("far,thin", [(400.0, 400.0), (1500.0, 20.0), (20000.0, 20000.0)])
def test_cube_faces(far, thin):
    """Triangles that cross the borders of the faces they are drawn on."""
    tl = [screen_tri(x, y, z, 1024, 1024) for x, y, z in triangles(300, 1024, 1024, far, thin, seed=8)]
    sc = tri_scene(tl, 64, 48, descs=TWO_SIDED,
                   lights=np.stack([S.make_light((0, 0, 0), radius=1e6, shadow=1),
                                    S.make_light((70, -40, 20), radius=1e6, shadow=1)]))
    gs = GpuScene(sc)
    gs.shadow_pass()
    dyn, _ = O.shadow(sc)
    assert (dyn != 0xFFFFFFFF).mean() > 0.01
    assert np.array_equal(gs.cubemaps()[:len(dyn)], dyn)
    gs.close()
