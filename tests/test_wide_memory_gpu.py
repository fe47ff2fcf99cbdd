"""Device memory is short: a call that fits beside the kd-trees alone gets the
wide tree's memory, and returns what it returns otherwise."""
import numpy as np
import pytest

from conftest import cuda_available
from yar_gb300 import native, scenes

pytestmark = pytest.mark.gpu

KERNELS = (native.TRAVERSAL_PERSISTENT_64, native.TRAVERSAL_PERSISTENT_128, native.TRAVERSAL_PER_RAY,
           native.TRAVERSAL_PER_RAY_VOTE)


@pytest.fixture(scope="module")
def torch_cuda():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import torch
    return torch


@pytest.fixture(scope="module")
def scene():
    s = scenes.large_scene(seed=1, width=256, height=256, spp=16, maxdepth=4, meshes=40)
    assert s.triangle_count > 800_000
    return s


def free_bytes(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


class Occupied:
    """All but `left` bytes of the device's free memory, in plain allocations."""

    def __init__(self, torch, left):
        self.torch = torch
        self.blocks = []
        size = 1 << 36
        while size >= 1 << 21:
            try:
                if free_bytes(torch) - size >= left:
                    self.blocks.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                    continue
            except torch.cuda.OutOfMemoryError:
                pass
            size >>= 1

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.blocks.clear()
        self.torch.cuda.empty_cache()


def with_context(kernel, s, use):
    ctx = native.Context(0, traversal_kernel=kernel)
    try:
        ctx.upload_scene(s)
        return use(ctx)
    finally:
        ctx.close()


def tree_bytes(torch, s):
    def used(kernel):
        before = free_bytes(torch)
        return with_context(kernel, s, lambda ctx: before - free_bytes(torch))
    used(native.TRAVERSAL_AUTO)
    return used(native.TRAVERSAL_AUTO) - used(native.TRAVERSAL_PER_RAY)


def test_render_gets_the_trees_memory(torch_cuda, scene):
    torch = torch_cuda
    tree = tree_bytes(torch, scene)
    assert tree > 100 << 20
    for kernel in KERNELS:  # (their local memory is allocated once per process)
        want = with_context(kernel, scene, lambda ctx: ctx.render(256, 256))
    need = []

    def measure(ctx):
        before = free_bytes(torch)
        ctx.render(256, 256)
        need.append(before - free_bytes(torch))
    with_context(native.TRAVERSAL_AUTO, scene, measure)

    def short(ctx):
        with Occupied(torch, need[0] - tree // 2):
            return [ctx.render(256, 256) for _ in range(2)]
    for img, stats in with_context(native.TRAVERSAL_AUTO, scene, short):
        assert img.tobytes() == want[0].tobytes()
        assert stats.variance == want[1].variance and stats.rays_closest == want[1].rays_closest


def test_host_cast_gets_the_trees_memory(torch_cuda, scene):
    torch = torch_cuda
    tree = tree_bytes(torch, scene)
    lo, hi = scenes.scene_box(scene)
    n = 1 << 22
    rays = scenes.random_rays(lo, hi, n, 71)
    for kernel in KERNELS:
        want = with_context(kernel, scene, lambda ctx: ctx.cast_closest(rays))
    staging = 52 * n  # rays and results

    def short(ctx):
        with Occupied(torch, staging - tree // 2):
            return ctx.cast_closest(rays)
    for g, w in zip(with_context(native.TRAVERSAL_AUTO, scene, short), want):
        assert g.tobytes() == w.tobytes()


def test_cast_without_memory_for_the_answers(torch_cuda):
    """The kd-tree answers; the tree stays for the next cast."""
    torch = torch_cuda
    s = scenes.raycast_scene(seed=2, grid=48, spheres=5, level=2)
    lo, hi = scenes.scene_box(s)
    n = 1 << 26
    few = torch.as_tensor(scenes.random_rays(lo, hi, 1 << 20, 72)).cuda()
    rays = few.repeat(n >> 20, 1)
    shadow = torch.zeros(n, dtype=torch.uint8, device="cuda")
    t = torch.zeros(n, dtype=torch.float32, device="cuda")
    prim, obj = torch.zeros((2, n), dtype=torch.int32, device="cuda")

    def cast(ctx):
        for out in (t, prim, obj, shadow):
            out.zero_()
        torch.cuda.synchronize()
        ctx.cast_closest_device(rays.data_ptr(), n, t.data_ptr(), prim.data_ptr(), obj.data_ptr())
        ctx.cast_any_device(rays.data_ptr(), n, shadow.data_ptr())
        return [x.cpu().numpy().tobytes() for x in (t, prim, obj, shadow)]
    want = with_context(native.TRAVERSAL_PERSISTENT_64, s, cast)

    def short(ctx):
        with Occupied(torch, 2 * n):  # of 4 n
            got = cast(ctx)
        assert ctx.traversal_kernels()["cast"] == [0, 0]
        return got, cast(ctx)
    got, later = with_context(native.TRAVERSAL_AUTO, s, short)
    assert got == want and later == want
