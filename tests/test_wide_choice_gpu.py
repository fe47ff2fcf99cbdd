"""Which scenes are cast through the wide tree, and what the library reports
about it.  A large enough cast times the kd-tree kernels of a scene without a
wide tree and reports the fastest; with one there is nothing to time and AUTO
(0) is reported, the option that selects the tree."""
import numpy as np
import pytest

from conftest import cuda_available, golden
from test_wide_gpu import assert_settled, probing_rays, soup
from yar_gb300 import native, scenes
from yar_gb300.scene import FlatScene

pytestmark = pytest.mark.gpu

TIMED_RAYS = 1 << 20  # a cast of this size times the kd-tree kernels


@pytest.fixture(autouse=True)
def needs_device():
    if not cuda_available():
        pytest.skip("no CUDA device")


def casts_through_wide_tree(s):
    ctx = native.Context(0)
    try:
        ctx.upload_scene(s)
        lo, hi = scenes.scene_box(s)
        rays = scenes.random_rays(lo, hi, TIMED_RAYS, 61)
        ctx.cast_closest(rays)
        ctx.cast_any(rays)
        kernels = ctx.traversal_kernels()["cast"]
    finally:
        ctx.close()
    assert (kernels[0] == 0) == (kernels[1] == 0), kernels
    return kernels[0] == 0


def test_reported_kernels_select_what_ran():
    """The wide tree is reported as AUTO, a timed kd-tree kernel as itself."""
    assert casts_through_wide_tree(soup(5000, 21))
    assert not casts_through_wide_tree(FlatScene.read(golden("transform_small.yfs")))
