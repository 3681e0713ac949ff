"""Launch shapes and scene forms that the traversal picks by size: short
streams and waves, and scenes that unroll to more placements than are laid
out."""
import numpy as np
import pytest

from psychopath_cpp_b200 import api, scenes
from psychopath_cpp_b200.scene import Assembly, Sphere
from tests import parity

pytestmark = pytest.mark.gpu
FIELDS = ("hit", "t", "uv", "p", "n", "dpdu", "backfacing", "offset", "space", "closure", "closure_color")


def equal(a, b):
    return all(np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f") for k in a)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1183, 1184, 2367, 2368, 9473, 37887, 37888])
def test_short_stream_is_the_stream_s_beginning(ctx, n):
    ctx.upload(scenes.plain_scene(3))
    rays = parity.random_rays(40000, (-6, -6, 0.01), (6, 6, 3), seed=5, occl_frac=0.3)
    whole = api.Tracer(ctx).trace(rays, fields=FIELDS + ("id",))
    part = api.Tracer(ctx).trace({k: v[:n] for k, v in rays.items()}, fields=FIELDS + ("id",))
    assert equal(part, {k: v[:n] for k, v in whole.items()})


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (17, 3, 1), (8, 8, 1), (13, 5, 2), (61, 47, 3), (160, 120, 2), (419, 313, 1),
                                     (311, 223, 3)])
def test_wave_length_does_not_change_the_film(ctx, w, h, spp):
    sc = scenes.plain_scene(4, res=(w, h), spp=spp)
    ctx.upload(sc)
    x, c = api.PathTraceIntegrator(ctx, w, h, spp, path_length=3).integrate()
    y, d = api.PathTraceIntegrator(ctx, w, h, spp, path_length=3, stream_paths=spp * max(1, w * h // 3)).integrate()
    assert np.array_equal(c, d) and np.array_equal(x, y)


def overgrown(sc):
    """`sc` with a far-away nest of some 270,000 assembly instances."""
    inner = Assembly()
    inner.add_object("s", Sphere([0.0, 0.0, 0.0], 0.5))
    inner.add_instance("s")
    for level in range(3):
        outer = Assembly()
        outer.add_assembly("in", inner)
        for k in range(65):
            outer.add_instance("in", [scenes.placement((0, 0, 1), 0.0, (2.0 * k, 0.0, 100.0 * level))])
        inner = outer
    sc.root.add_assembly("nest", inner)
    sc.root.add_instance("nest", [scenes.placement((0, 0, 1), 0.0, (1e5, 1e5, 1e5))])
    return sc


@pytest.mark.parametrize("seed", [1, 2])
def test_scene_without_placements_gives_the_same_hits(ctx, seed):
    """A scene past the placements' limit keeps a level stack per ray; with
    the nest out of every ray's way its hits and its film are those of the
    scene without the nest."""
    make = lambda: scenes.many_light_scene(seed, res=(48, 27), spp=2, n_patches=40, n_groups=20, n_lights=30)
    rays = parity.random_rays(20000, (-4, -4, -0.5), (4, 4, 5), seed=seed, occl_frac=0.3)
    got = []
    for sc in (make(), overgrown(make())):
        ctx.upload(sc)
        hits = api.Tracer(ctx).trace(rays, fields=FIELDS)
        film, counts = api.PathTraceIntegrator(ctx, 48, 27, 2, path_length=4).integrate()
        got.append((hits, film, counts))
    assert 0 < got[0][0]["hit"].sum() < len(rays["time"])
    assert equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_light_sample_rows_match_the_device_form(ctx, n):
    """psy_light_sample_rows (host rows) against psy_light_sample (device
    arrays) on the same queries."""
    import ctypes as C

    import torch

    from psychopath_cpp_b200 import _abi
    ctx.upload(scenes.batch_scene(5, (64, 64), 1, 20, 37))
    rng = np.random.default_rng(n)
    q = np.zeros((n, 15), np.float32)
    q[:, 0:3] = rng.random((n, 3))
    q[:, 3:6] = rng.uniform(-4, 4, (n, 3))
    for k in (6, 9):
        v = rng.normal(size=(n, 3))
        q[:, k:k + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    q[:, 12] = rng.uniform(380, 700, n)
    q[:, 13] = rng.random(n)
    rows, ids = api.LightTree(ctx).sample(q)
    cols = [torch.from_numpy(np.ascontiguousarray(q[:, c])).cuda()
            for c in (0, 1, 2, slice(3, 6), slice(6, 9), slice(9, 12), 12, 13)]
    out = [torch.zeros(s, dtype=t, device="cuda") for s, t in
           (((n, 3), torch.float32), ((n, 4), torch.float32), (n, torch.float32), (n, torch.float32), (n, torch.int64))]
    qs = _abi.LightQuerySoA(*[C.c_void_p(t.data_ptr()) for t in cols])
    ss = _abi.LightSampleSoA(*[C.c_void_p(t.data_ptr()) for t in out])
    ctx.check(ctx.L.psy_light_sample(ctx.h, C.byref(qs), n, C.byref(ss), None))
    ctx.sync()
    want = np.zeros((n, 14), np.float32)
    want[:, 0:3], want[:, 3:7] = out[0].cpu().numpy(), out[1].cpu().numpy()
    want[:, 7], want[:, 8], want[:, 9] = q[:, 12], out[2].cpu().numpy(), out[3].cpu().numpy()
    assert np.array_equal(rows, want) and np.array_equal(ids, out[4].cpu().numpy().view(np.uint64))


def test_batch_with_two_waves_in_flight_equals_plain_renders(ctx):
    entries = []
    for k, (w, h, spp) in enumerate([(301, 157, 2), (64, 48, 5), (233, 129, 3)]):
        c = api.Context(0)
        c.upload(scenes.batch_scene(k, (w, h), spp, 60 + 40 * k, 3 + k))
        entries.append({"scene": c, "width": w, "height": h, "spp": spp, "seed": 7 + k})
    b = api.BatchRenderer(ctx, entries)
    assert b.paths >= 1 << 17
    b.render()
    for e, (x, c) in zip(entries, b.images()):
        y, d = api.PathTraceIntegrator(e["scene"], e["width"], e["height"], e["spp"], seed=e["seed"],
                                       stream_paths=4096).integrate()
        assert np.array_equal(c, d) and np.array_equal(x, y)


def test_adjoint_with_two_waves_in_flight(ctx):
    """The gradient does not depend on the waves but for the order of its
    32-bit sums: at most some hundred blocks' sums are added to a parameter in
    either run, each rounding by half an ulp of the running total."""
    import torch
    w, h, spp = 256, 192, 4
    sc = scenes.adjoint_scene(2, res=(w, h), spp=spp)
    ctx.upload(sc)
    shaders, objects, ns, no = api.flat_indices(sc)
    sp, op, count = np.full(ns, -1, np.int32), np.full(no, -1, np.int32), 0
    for name, sh in sc.root.shaders.items():
        if name.startswith("mat"):
            sp[shaders[id(sh)]] = count
            count += 4
    for name in sc.root.objects:
        if name.startswith("light"):
            op[objects[(0, name)]] = count
            count += 1
    params = torch.full((count,), 0.6, device="cuda")
    dl = torch.rand(h * w * 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    g = [api.DiffRenderer(ctx, w, h, spp, sp, op, count, stream_paths=s).adjoint(params, dl).double()
         for s in (0, 50000)]
    assert w * h * spp >= 1 << 17
    # 8 launches of at most 3 * 148 blocks, twice: 7104 additions of 2^-24
    bound = 7104 * 2.0 ** -24
    assert torch.all((g[0] - g[1]).abs() <= bound * g[1].abs().clamp_min(float(g[1].abs().max()) * 1e-3))


@pytest.mark.parametrize("zeros", [1, 2])
@pytest.mark.parametrize("name", ["plain", "motion"])
def test_rays_with_zero_components_match_the_oracle(ctx, name, zeros):
    """Rays whose slab tests can meet 0 * inf (direction components of zero)
    take the reference's own minima and maxima, out of line; the others single
    instructions.  Both against the plain-C oracle."""
    from oracle import port
    sc = {"plain": scenes.plain_scene, "motion": scenes.motion_patch_scene}[name](6)
    rays = parity.random_rays(3000, (-4, -4, 0.01), (4, 4, 3), seed=zeros, occl_frac=0.3)
    rng = np.random.default_rng(zeros)
    k = np.arange(0, 3000, 2)  # every other ray
    for _ in range(zeros):
        rays["d"][k, rng.integers(0, 3, k.size)] = 0.0
    rays["d"][np.all(rays["d"] == 0.0, axis=1), 2] = -1.0
    ctx.upload(sc)
    mine = api.Tracer(ctx).trace(rays, fields=("hit", "id", "t", "uv", "closure"))
    ref = port.trace(sc, rays)
    patch = (ref["uv"][:, 0] != 0) & (mine["closure"] == 1)
    assert 100 < int(mine["hit"].sum()) < 3000
    parity.assert_parity(parity.compare_trace(ref, mine, rays["type"], uv_mask=patch))
