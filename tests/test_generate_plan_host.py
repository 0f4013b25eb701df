"""How a generation step is split over clusters (generate_plan.hpp), compiled for the host: as few sequences per cluster as leave one round,
and never more clusters than the form that is taken has room for."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("plan") / "libplan_host.so")
    src = os.path.join(ROOT, "tests", "host_harness", "plan_host.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", src, "-o", out], check=True)
    lib = C.CDLL(out)

    def run(batch, any_room, own_room, divides=16, fit_group=4):
        got = np.zeros(4, np.uint32)
        lib.plan_host(C.c_uint64(batch), 16, 4, C.c_uint32(divides), C.c_uint32(fit_group), any_room, own_room, C.c_void_p(got.ctypes.data))
        return dict(zip(("cluster", "group", "grid", "asked"), (int(x) for x in got)))

    return run


@pytest.mark.parametrize("batch,cluster,group,grid", [(1, 16, 1, 16), (9, 16, 1, 144), (10, 16, 2, 80), (36, 16, 4, 144), (37, 8, 4, 80), (64, 8, 4, 128),
                                                      (72, 8, 4, 144), (73, 4, 2, 148), (592, 1, 4, 148), (1000, 1, 4, 148)])
def test_one_round_with_the_most_ctas_per_cluster(plan, batch, cluster, group, grid):
    assert plan(batch, 148, 148) == {"cluster": cluster, "group": group, "grid": grid, "asked": 1}


@pytest.mark.parametrize("batch", [1, 9, 40, 64, 100, 592, 1000])
@pytest.mark.parametrize("any_room,own_room", [(148, 74), (296, 148), (148, 296), (148, 33)])
def test_the_form_that_is_taken_has_the_last_word(plan, batch, any_room, own_room):
    p, q = plan(batch, any_room, own_room), plan(batch, any_room, any_room)
    assert (p["cluster"], p["group"], p["asked"]) == (q["cluster"], q["group"], 1)
    want = (batch + p["group"] - 1) // p["group"]
    assert p["grid"] == min(want, own_room // p["cluster"]) * p["cluster"] <= own_room


def test_no_room_means_no_kernel(plan):
    assert plan(8, 148, 8)["grid"] == 0                       # the form taken has none: clusters of 16 on 8 CTAs
    assert plan(8, 0, 148) == {"cluster": 0, "group": 1, "grid": 0, "asked": 0}
    assert plan(8, 148, 148, fit_group=0) == {"cluster": 0, "group": 1, "grid": 0, "asked": 0}
