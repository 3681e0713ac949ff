"""Bounding boxes that the traversal's plain node test does not cover:
inverted ones (a radius below zero).  The reference takes the near plane of an
axis by the ray's sign (basics/bbox.hpp:566-595), so no ray hits them.  Times
outside the samples, which can invert a box too."""
import numpy as np
import pytest

from psychopath_cpp_b200 import api, scenes
from psychopath_cpp_b200.scene import Sphere, SphereLight
from tests import parity

pytestmark = pytest.mark.gpu
FIELDS = ("hit", "id", "t", "uv", "p", "n", "closure")


def trace(ctx, scene, rays, gpu_bvh):
    ctx.upload(scene, gpu_bvh=gpu_bvh)
    return api.Tracer(ctx).trace(rays, fields=FIELDS)


def equal(a, b, rays):
    # (which of its blockers ends a shadow ray depends on the tree)
    closest = rays["type"] != 32
    return (np.array_equal(a["id"][closest], b["id"][closest])
            and all(np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f") for k in a if k != "id"))


@pytest.mark.parametrize("gpu_bvh", [False, True])
@pytest.mark.parametrize("zeros", [False, True])
def test_spheres_of_negative_radius_are_not_hit(ctx, gpu_bvh, zeros):
    rays = parity.random_rays(20000, (-6, -6, 0.01), (6, 6, 3), seed=3, occl_frac=0.3)
    if zeros:
        rays["d"][::2, 1] = 0.0
    sc = scenes.plain_scene(5)
    want = trace(ctx, sc, rays, gpu_bvh)
    rng = np.random.default_rng(1)
    for k in range(40):  # (the same number of id bits: 66 and 106 instances)
        sc.root.add_object("neg%d" % k, Sphere(rng.uniform((-5, -5, 0), (5, 5, 2)), -rng.uniform(0.2, 0.6)))
        sc.root.add_instance("neg%d" % k, shader="mat0")
    got = trace(ctx, sc, rays, gpu_bvh)
    assert 1000 < int(want["hit"].sum()) < 20000
    assert equal(got, want, rays)


def test_light_whose_radius_changes_sign(ctx):
    """Two time samples of a light, of which the first one's box is inverted:
    hit when the radius at the ray's time is above zero, else not."""
    rays = parity.random_rays(20000, (-6, -6, 0.01), (6, 6, 3), seed=4)
    sc = scenes.plain_scene(6)
    plain = scenes.plain_scene(6)
    for s, radii in ((sc, [-0.5, 0.5]), (plain, [0.25, 0.25])):
        s.root.add_object("big", SphereLight([[0.0, 0.0, 1.0]], radii, [[1.0] * 3]))
        s.root.add_instance("big")
    rays["time"][:] = 0.75  # the radius is 0.25, without rounding
    assert equal(trace(ctx, sc, rays, False), trace(ctx, plain, rays, False), rays)
    rays["time"][:] = 0.25
    got, want = trace(ctx, sc, rays, False), trace(ctx, scenes.plain_scene(6), rays, False)
    assert equal(got, want, rays)


@pytest.mark.parametrize("time,hits", [(-0.9, False), (-0.75, False), (0.5, True)])
def test_boxes_extrapolated_before_the_first_sample(ctx, time, hits):
    """Lights whose radius, taken on to a time before the first sample, is
    below zero: their boxes are inverted at that time."""
    rays = parity.random_rays(20000, (-6, -6, 0.01), (6, 6, 3), seed=5, occl_frac=0.3)
    rays["time"][:] = time
    rng = np.random.default_rng(2)
    sc = scenes.Scene(name="growing")
    for k in range(30):
        sc.root.add_object("grow%d" % k, SphereLight([rng.uniform((-5, -5, 0), (5, 5, 2))], [0.5, 1.5], [[1.0] * 3]))
        sc.root.add_instance("grow%d" % k)
    assert bool(trace(ctx, sc, rays, False)["hit"].any()) == hits


@pytest.mark.parametrize("scene", ["motion", "instanced"])
def test_times_far_outside_the_samples(ctx, scene):
    """Nothing outside the samples is read: the call ends without an error and
    hits nothing that is not there at any time."""
    sc = scenes.motion_patch_scene(2) if scene == "motion" else scenes.many_light_scene(4, n_patches=60, n_groups=30, n_lights=50)
    rays = parity.random_rays(20000, (-4, -4, 0.01), (4, 4, 3), seed=6, occl_frac=0.3)
    rays["time"][:] = np.random.default_rng(1).choice(np.array([-1.0, -1.5, -3.0, 1.0, 2.5, 7.0], np.float32), 20000)
    got = trace(ctx, sc, rays, False)
    assert 1000 < int(got["hit"].sum()) < 20000
    assert np.all(got["t"][(got["hit"] == 1) & (rays["type"] != 32)] > 0.0)
