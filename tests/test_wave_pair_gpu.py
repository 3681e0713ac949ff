"""Renders whose paths run as two waves in flight, where the second wave's
buffers may not or cannot be allocated: while the caller's stream is captured,
and without the memory for it."""
import pytest

from psychopath_cpp_b200 import api, scenes

pytestmark = pytest.mark.gpu
W, H, SPP = 419, 313, 2  # 262,294 paths


@pytest.fixture
def fresh():
    c = api.Context(0)
    c.upload(scenes.plain_scene(3, res=(W, H), spp=SPP))
    yield c
    c.close()


def film(torch):
    return torch.zeros(H * W * 3, device="cuda"), torch.zeros(H * W, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("warm", [W * H * SPP, 0])
def test_capture_with_one_or_two_waves_of_buffers(fresh, warm):
    """A context that has rendered in one wave (warm) or in two can be captured
    rendering by itself: no allocation then."""
    import torch
    want, counts = film(torch)
    api.PathTraceIntegrator(fresh, W, H, SPP, stream_paths=warm).integrate_device(want, counts, with_stats=True)
    x, c = film(torch)
    auto = api.PathTraceIntegrator(fresh, W, H, SPP)
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        auto.integrate_device(x, c, s.cuda_stream, with_stats=False)
    assert not x.any()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want) and torch.equal(c, counts)


def test_without_memory_for_a_second_wave(fresh):
    """Memory for one wave of half the paths, not for two: the render runs its
    waves one after another."""
    import torch
    want, counts = film(torch)
    api.PathTraceIntegrator(fresh, W, H, SPP, stream_paths=4096).integrate_device(want, counts, with_stats=True)
    x, c = film(torch)
    auto = api.PathTraceIntegrator(fresh, W, H, SPP)
    torch.cuda.synchronize()
    half = W * H * SPP // 2 * 357  # bytes of such a wave
    held = []
    try:
        for size in (1 << 30, 1 << 26, 1 << 24):  # (torch takes each as it is)
            while torch.cuda.mem_get_info()[0] > size + 3 * half // 2:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        auto.integrate_device(x, c, with_stats=True)
        waves = auto.stats.waves
    finally:
        del held
        torch.cuda.empty_cache()
    assert waves == 2 and torch.equal(x, want) and torch.equal(c, counts)
