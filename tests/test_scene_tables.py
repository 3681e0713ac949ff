"""The unrolled assembly instances of a scene (CPU): their contents, and that
laying them out costs time by the entry, not by the object of every placed
assembly."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "psychopath_cpp_b200", "csrc")


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tables") / "libscene_host.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I" + CSRC,
                    "-I" + os.path.join(os.path.dirname(HERE), "include"), os.path.join(HERE, "scene_host.cpp"),
                    os.path.join(CSRC, "scene_build.cpp"), os.path.join(CSRC, "host_cpu.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.place_tables.restype = C.c_double

    def f(objects, placed, limit=1 << 18):
        n, right = C.c_int(), C.c_int()
        s = min(L.place_tables(objects, placed, limit, C.byref(n), C.byref(right)) for _ in range(3))
        return s, n.value, bool(right.value)
    return f


@pytest.mark.parametrize("objects,placed", [(1, 1), (5, 7), (1, 4095), (100, 1000)])
def test_entries(tables, objects, placed):
    assert tables(objects, placed)[1:] == (placed + 1, True)


@pytest.mark.parametrize("limit,entries", [(8, 8), (7, 0), (9, 8)])
def test_scenes_past_the_limit_have_none(tables, limit, entries):
    assert tables(3, 7, limit)[1:] == (entries, True)


@pytest.mark.parametrize("placed,entries", [(50000, 50001), (200000, 200001), (300000, 0)])
def test_time_does_not_grow_with_the_objects_of_a_placed_assembly(tables, placed, entries):
    """20,000 objects in the assembly: 1e9 and 4e9 steps if every placement
    passed over them, some seconds."""
    small, n, _ = tables(1, placed)
    large, m, right = tables(20000, placed)
    assert n == m == entries and right
    assert large < 5 * small + 0.1
