"""The waves of a batch (CPU): what the caller, the autotuner or neither asks
for, and that they hold the paths wanted within the paths there are."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "psychopath_cpp_b200", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "libplan_host.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I" + CSRC, os.path.join(HERE, "plan_host.cpp"),
                    "-o", so], check=True)
    L = C.CDLL(so)

    def f(total, spp, stream_paths=0, tuned=0):
        p = C.c_uint64()
        pair = L.batch_wave(C.c_uint64(total), C.c_uint32(spp), C.c_uint32(stream_paths), C.c_uint32(tuned), C.byref(p))
        return p.value, bool(pair)
    return f


@pytest.mark.parametrize("total", [1, 1000, (1 << 17) - 1, 1 << 17, 300001, 1 << 22, 10 ** 9])
@pytest.mark.parametrize("spp", [1, 7, 128])
def test_plans(plan, total, spp):
    spp = min(spp, total)
    for lg in range(10, 27):
        n = 1 << lg
        # the caller's number: one wave after another
        assert plan(total, spp, stream_paths=n, tuned=1 << 20) == (min(max(n, spp), total), False)
        # the autotuner's number, which it times in the same form: in flight
        paths, pair = plan(total, spp, tuned=n)
        assert pair == (min(n, total) >= 1 << 17)
        want = min(n, total)
        assert paths == min(total, (want + 1) // 2 + spp if pair else max(want, spp))
    assert plan(total, spp) == plan(total, spp, tuned=1 << 22)
