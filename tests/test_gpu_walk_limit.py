"""A walk that ends on its step budget is reported against the budget it was
held to: a batch's walks share the smallest of their scenes' budgets, which may
be less than the walk's own scene's."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from hydra_lotus_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def driver(cuda, tmp_path_factory):
    lib = os.path.join(tmp_path_factory.mktemp("walk"), "libwalk_limit.so")
    subprocess.run(["nvcc"] + build.ARCH + build.FLAGS + ["--fmad=false", "-shared", os.path.join(HERE, "walk_limit.cu"),
                                                          "-o", lib], check=True)
    return C.CDLL(lib)


def walk(driver, nodes, scene_limit, limit, round_):
    words = np.zeros(3, dtype=np.uint32)
    assert driver.walk_chain(nodes, C.c_uint(scene_limit), C.c_uint(limit), round_,
                             words.ctypes.data_as(C.c_void_p)) == 0
    return [int(w) for w in words]


@pytest.mark.parametrize("nodes,scene_limit,limit,cut", [
    (8, 1000, 1000, False),  # far below both
    (8, 1000, 4, True),      # cut by the smaller budget of another scene
    (8, 1000, 8, True),      # the budget used up by the last step
    (8, 1000, 9, False),
    (8, 4, 1000, False),     # the scene's own budget is not the walk's
    (1, 1000, 1, True),
    (32, 1000, 1, True)])
def test_cut_walk_is_reported(driver, nodes, scene_limit, limit, cut):
    failed, causes, steps = walk(driver, nodes, scene_limit, limit, 1)
    assert steps == min(nodes, limit)
    assert failed == (1 if cut else 0)
    assert (causes != 0) == cut


@pytest.mark.parametrize("limit,cut", [(4, 1), (8, 1), (9, 0)])
def test_traverse_is_held_to_the_scene_budget(driver, limit, cut):
    assert walk(driver, 8, limit, 0, 0)[0] == cut
