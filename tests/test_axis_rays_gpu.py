"""Rays along an axis and patches with huge coordinates: what the bisection
tests with the reference's own minima and maxima, out of line and, in a render,
a limited number of steps at a time."""
import numpy as np
import pytest

from psychopath_cpp_b200 import api, scenes
from psychopath_cpp_b200.scene import BicubicPatch, BilinearPatch, Camera, Sphere, SurfaceShader
from tests import parity

pytestmark = pytest.mark.gpu


def huge_scene(kind):
    """A ground patch far past the coordinates whose sums are known to stay
    finite, and a sphere on it."""
    h = 2e37
    sc = scenes.Scene(name="huge")
    sc.root.add_shader("m", SurfaceShader("Lambert", [0.5] * 3))
    if kind == "bilinear":
        sc.root.add_object("ground", BilinearPatch([[-h, -h, 0], [h, -h, 0], [-h, h, 0], [h, h, 0]]))
    else:
        k = np.linspace(-h, h, 4)
        sc.root.add_object("ground", BicubicPatch(np.stack([[[x, y, 0.0] for x in k] for y in k]).reshape(16, 3)))
    sc.root.add_object("ball", Sphere([0.0, 0.0, 1.0], 0.5))
    for name in ("ground", "ball"):
        sc.root.add_instance(name, shader="m")
    return sc


def down(rays):
    rays["d"][:] = (0.0, 0.0, -1.0)
    return rays


@pytest.mark.parametrize("width", [0.0, 0.05])
@pytest.mark.parametrize("name", ["motion", "heightfield", "bilinear", "bicubic"])
def test_streams_straight_down_match_the_oracle(ctx, name, width):
    from oracle import port
    sc = {"motion": lambda: scenes.motion_patch_scene(6), "heightfield": lambda: scenes.heightfield_scene(8, seed=2),
          "bilinear": lambda: huge_scene("bilinear"), "bicubic": lambda: huge_scene("bicubic")}[name]()
    lo, hi = ((0, 0, 1), (8, 8, 4)) if name == "heightfield" else ((-3, -3, 0.5), (3, 3, 4))
    rays = down(parity.random_rays(1500, lo, hi, seed=8, occl_frac=0.3, width=width))
    if name in ("bilinear", "bicubic"):
        rays["d"][::3] = parity.random_rays(500, lo, hi, seed=9)["d"]  # (the patch is odd for every ray)
    ctx.upload(sc)
    mine = api.Tracer(ctx).trace(rays, fields=("hit", "id", "t", "uv", "closure"))
    ref = port.trace(sc, rays)
    patch = (ref["uv"][:, 0] != 0) & (mine["closure"] == 1)
    assert int(mine["hit"].sum()) > 300
    parity.assert_parity(parity.compare_trace(ref, mine, rays["type"], uv_mask=patch))


@pytest.mark.parametrize("scene", ["bilinear", "motion"])
def test_camera_rays_straight_down(ctx, scene):
    """A camera without an angle of view that moves sideways over the scene:
    all its rays are straight down.  Against the same rays 1e-7 off the axis:
    the hits move by some 1e-5 (the size the patches are diced to), so the
    light that arrives changes by about 1e-4, but for the few samples whose
    shadow ray passes an edge."""
    w, h = 96, 64
    film = []
    for tilt in (0.0, 1e-7):
        sc = scenes.motion_patch_scene(3) if scene == "motion" else scenes.plain_scene(3, light_radius=0.1)
        at = []
        for x in (-4.0, 4.0):
            m = np.diag([1.0, -1.0, -1.0, 1.0])
            m[2, :2] = tilt
            m[3, :3] = (x, 0.37, 20.0)
            at.append(m)
        sc.camera = Camera(transforms=at, fovs=[0.0])
        ctx.upload(sc)
        film.append(api.PathTraceIntegrator(ctx, w, h, 1, path_length=1).integrate()[0][..., 1])
    a, b = film
    lit = (a > 0) & (b > 0)
    assert lit.sum() > 0.5 * w * h
    assert np.mean((a > 0) == (b > 0)) > 0.98
    assert np.mean(np.abs(a[lit] / b[lit] - 1.0) < 1e-3) > 0.98
