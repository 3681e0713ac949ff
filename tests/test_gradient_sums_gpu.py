"""The adjoint's sums: a block gathers its gradient in 64 bits, with more
parameters in 32, with more still it adds to the output itself.

The gradient is linear in dL/dfilm, so the sum in 64 bits of adjoints whose
dL/dfilm is cut to a few rows each is a gradient with little rounding: each
part rounds as its own small total.  A 32-bit sum of n terms of one sign has a
random error of about sqrt(n / 3) * 2^-24 / 2 of it; five times that is
allowed."""
import numpy as np
import pytest

from psychopath_cpp_b200 import api, scenes

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24


def problem(ctx, w, h, spp):
    sc = scenes.adjoint_scene(2, res=(w, h), spp=spp)
    ctx.upload(sc)
    shaders, objects, ns, no = api.flat_indices(sc)
    sp, op, count = np.full(ns, -1, np.int32), np.full(no, -1, np.int32), 0
    for name, sh in sc.root.shaders.items():
        if name.startswith("mat"):
            sp[shaders[id(sh)]] = count
            count += 4
    lights = []
    for name in sc.root.objects:
        if name.startswith("light"):
            op[objects[(0, name)]] = count
            lights.append(count)
            count += 1
    return sp, op, count, lights


def gradients(ctx, w, h, spp, counts, parts):
    """The gradients with each of the parameter counts (those past the first
    not used), and the 64-bit sum of `parts` adjoints."""
    import torch
    sp, op, used, lights = problem(ctx, w, h, spp)
    dl = torch.rand(h, w * 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out = []
    for n in counts:
        params = torch.full((n or used,), 0.6, device="cuda")
        r = api.DiffRenderer(ctx, w, h, spp, sp, op, n or used)
        out.append(r.adjoint(params, dl.reshape(-1)).double()[:used].cpu().numpy())
    params = torch.full((used,), 0.6, device="cuda")
    r = api.DiffRenderer(ctx, w, h, spp, sp, op, used)
    exact = torch.zeros(used, dtype=torch.float64, device="cuda")
    for k in range(parts):
        rows = torch.zeros_like(dl)
        rows[k::parts] = dl[k::parts]
        exact += r.adjoint(params, rows.reshape(-1)).double()
    return out, exact.cpu().numpy(), lights


@pytest.mark.parametrize("count", [4096, 4097, 8192, 8193])
def test_every_form_of_the_sum(ctx, count):
    """At the limits of the three forms: 4,096 parameters in 64 bits, 4,097
    and 8,192 in 32, 8,193 without shared memory."""
    w, h, spp = 128, 96, 16
    (g,), exact, _ = gradients(ctx, w, h, spp, [count], 8)
    n = w * h * spp * 4  # a path adds at most once a vertex to a parameter
    bound = 5 * np.sqrt(n / 3.0) * ULP / 2
    assert np.mean(exact != 0.0) > 0.8
    assert np.all(np.abs(g - exact) <= bound * np.abs(exact).max())


def test_block_sums_of_many_terms(ctx):
    """4M paths: the emission gradients (terms of one sign) are as exact as
    adding the blocks' 64-bit sums in 32 bits lets them be: two waves of four
    shading launches and the last shadow rays', of at most 3 blocks an SM."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    (g,), exact, lights = gradients(ctx, 256, 256, 64, [0], 32)
    bound = 5 * np.sqrt(2 * 5 * 3 * sms / 3.0) * ULP / 2
    assert np.all(np.abs(g[lights] - exact[lights]) <= bound * exact[lights])
