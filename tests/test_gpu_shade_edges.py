"""kernel3 at the edges of its arithmetic, against the oracle."""
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


def compare(sc):
    """The scene's first view by the GPU and by the oracle; RGBA within 1/255."""
    gs = GpuScene(sc)
    got = gs.render(sc.cameras[0], sc.views[0]).numpy()
    gs.close()
    ref = O.render(sc, O.build_textures(sc.tex_sizes, sc.tex_pixels), sc.cameras[0], sc.views[0])
    assert np.array_equal(got["depth"], ref["depth"]) and np.array_equal(got["id"], ref["id"])
    d = np.abs(got["rgba"].astype(int) - ref["rgba"].astype(int))
    assert d.max() <= 1, f"{int((d > 1).any(-1).sum())} pixels off, by up to {int(d.max())}"
    return ref["rgba"]


def plane(w, h, z0, z1, **kw):
    """A quad over the whole view, z0 at its left edge and z1 at its right, facing the eye."""
    lo, hi = (-10, -10), (w + 10, h + 10)
    return tri_scene([screen_tri([lo[0], lo[0], hi[0]], [lo[1], hi[1], lo[1]], [z0, z0, z1], w, h),
                      screen_tri([hi[0], lo[0], hi[0]], [lo[1], hi[1], hi[1]], [z1, z0, z1], w, h)], w, h, **kw)


@pytest.mark.parametrize("specular", [0.9, 0.95])
def test_outline_over_subnormal_colour(specular):
    """A channel that only the foot of a highlight reaches, far below the smallest normal float: the outline added after
    the output gamma shows there all the same."""
    w, h = 400, 300
    d = S.make_descriptor(tid=0, feature_flag=S.FLAG_OUTLINE, specular=specular)
    sc = plane(w, h, 2000.0, 60000.0, descs=np.stack([d]),
               lights=np.stack([S.make_light((60000.0, -3000.0, 2000.0), radius=200000.0, brightness=4.0)]))
    sc.tex_pixels = [np.tile(np.array([255, 0, 0, 255], np.uint8), (64, 64, 1))]
    sc.views = [S.make_view(w, h, 90.0, flags=S.VIEW_OUTLINE)]
    rgba = compare(sc)
    assert (rgba[..., 1] > 3).mean() > 0.5  # the outline, in a channel that the texture leaves at 0


@pytest.mark.parametrize("pos,radius", [((0.0, 0.0, -3.0e19), 2.0e19), ((2.0e20, 1.0e20, 0.0), 1.0e20),
                                        ((0.0, 5.0e18, -5.0e18), 1.0e19), ((0.0, -1.0e25, 0.0), 3.0e30),
                                        ((0.0, 1.0e19, -1.0e19), -1.0e19), ((3.0e20, 0.0, 0.0), -1.0e19)])
@pytest.mark.parametrize("shadow", [0, 1])
def test_lights_farther_than_a_square_can_hold(pos, radius, shadow):
    """Distances whose squares overflow, or come close, are as dark as the oracle has them."""
    w, h = 200, 150
    sc = plane(w, h, 300.0, 900.0, descs=np.stack([S.make_descriptor(tid=0)]),
               lights=np.stack([S.make_light(pos, radius=radius, brightness=1.0, shadow=shadow),
                                S.make_light((0.0, 0.0, 10.0), radius=600.0)]))
    compare(sc)


@pytest.mark.parametrize("radius", [0.0, -1000.0])
def test_dark_lights_opposite_the_eye(radius):
    """Lights that add nothing, right behind the surface as the eye sees it, leave another light's highlight alone."""
    w, h = 300, 300
    rng = np.random.default_rng(2)
    dark = [S.make_light((*rng.uniform(-3e4, 3e4, 2), 4.0e6), radius=radius) for _ in range(60)]
    sc = plane(w, h, 900.0, 900.0, lights=np.stack([S.make_light((0.0, 0.0, 10.0), radius=4000.0, brightness=8.0)] + dark))
    sc.tex_pixels = [np.tile(np.array([0, 0, 0, 255], np.uint8), (64, 64, 1))]
    sc.views = [S.make_view(w, h, 1.0)]
    for t in sc.tris:  # screen_tri laid them out for 90 degrees
        for v in t["vertices"]:
            v["pos"][:2] *= w / 2.0 / O.fov_const(1.0, w)
    rgba = compare(sc)
    assert (rgba[..., :3] > 50).all(-1).mean() > 0.9
