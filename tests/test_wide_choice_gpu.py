"""Which scenes are cast through the wide tree, and what the library reports
about it.  A large enough cast times the kd-tree kernels of a scene without a
wide tree and reports the fastest; with one there is nothing to time and AUTO
(0) is reported, the option that selects the tree."""
import numpy as np
import pytest

from conftest import cuda_available, golden
from test_wide_gpu import assert_settled, probing_rays, soup
from yar_gb300 import native, scenes
from yar_gb300.scene import FlatScene, Mesh, make_object

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


def flat_scene(triangles):
    """One untransformed mesh of the triangles [n, 3, 3]."""
    s = FlatScene()
    p = np.asarray(triangles, np.float32)
    s.meshes.append(Mesh(p.reshape(-1, 3), np.arange(3 * len(p)).reshape(-1, 3)))
    m = np.eye(3, 4, dtype=np.float32).ravel()
    s.objects = np.array([make_object(0, m, m)])
    s.build_kdtrees(1)
    return s


def unit_cube():
    c = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64)
    quads = [(0, 1, 3, 2), (4, 5, 7, 6), (0, 1, 5, 4), (2, 3, 7, 6), (0, 2, 6, 4), (1, 3, 7, 5)]
    return np.array([[c[q[0]], c[q[k]], c[q[k + 1]]] for q in quads for k in (1, 2)])


def fence():  # 2,000 equal cubes in a row
    return unit_cube()[None] + 2.0 * np.arange(2000)[:, None, None, None] * np.array([1.0, 0, 0])


def strip():  # 10,000 equal cells of a plane in a row
    cell = np.array([[[0, 0, 0], [1, 0, 0], [1, 1, 0]], [[0, 0, 0], [1, 1, 0], [0, 1, 0]]], np.float64)
    return cell[None] + np.arange(10000)[:, None, None, None] * np.array([1.0, 0, 0])


def copies():  # 1,500 triangles of one box among random ones
    rng = np.random.default_rng(31)
    p = rng.random((20000, 1, 3)) + 0.02 * (rng.random((20000, 3, 3)) - 0.5)
    p[7000:8500] = p[7000]
    p[7000:8500, 1, 2] += np.linspace(0, 1, 1500) * (p[7000, 2, 2] - p[7000, 1, 2])
    return p


def growing():  # each half a percent larger than the one before it and past its end
    k = 1.005 ** np.arange(3000)
    base = np.array([[0, 0, 0], [1, 0, 0.2], [0.3, 1, 0.4]])
    return k[:, None, None] * base + 210.0 * k[:, None, None] * np.array([1.0, 0, 0])


@pytest.mark.parametrize("make", [fence, strip, copies, growing])
def test_equal_and_growing_boxes(make):
    """Neighbours of equal area, and boxes that grow along the builder's order,
    above and below the cluster count that one block finishes: the tree is
    built, and its casts are the kd-tree's."""
    s = flat_scene(make().reshape(-1, 3, 3))
    assert casts_through_wide_tree(s)
    assert_settled(s, probing_rays(s, 32768, 32))
    small = flat_scene(make().reshape(-1, 3, 3)[:1000])
    assert casts_through_wide_tree(small)
    assert_settled(small, probing_rays(small, 16384, 33))


def test_launches_of_a_planar_scene():
    """Renders of a scene of tessellated planes walk the kd-tree, one kernel a
    cast: as many launches as with that kernel fixed, the same image."""
    torch = pytest.importorskip("torch")
    s = scenes.hard_lighting_room(cells=64)  # 49,000 triangles of axis-parallel planes
    s.config["render_region"] = (0, 0, 64, 64)
    got = []
    for kernel in (native.TRAVERSAL_AUTO, native.TRAVERSAL_PER_RAY):
        ctx = native.Context(0, traversal_kernel=kernel)
        try:
            ctx.upload_scene(s)
            assert ctx.traversal_kernels()["render_closest"] == [native.TRAVERSAL_PER_RAY] * 5
            ctx.render(64, 64)
            img, stats = ctx.render(64, 64)  # the second one: bounces driven from the device
            out = torch.zeros((64, 64, 3), dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            static = ctx.render_static(out.data_ptr())
            got.append((img.tobytes(), stats.kernel_launches, static.kernel_launches))
        finally:
            ctx.close()
    assert got[0] == got[1]


def moved(s, linear):
    """The scene with its second object under one more linear part."""
    o = s.objects[1]
    m = np.asarray(o["object_to_world"], np.float64).reshape(3, 4)
    m = np.concatenate([linear @ m[:, :3], m[:, 3:]], axis=1)
    inv = np.linalg.inv(np.concatenate([m, [[0, 0, 0, 1]]]))[:3]
    s.objects[1] = make_object(1, m.astype(np.float32).ravel(), inv.astype(np.float32).ravel())
    s.build_kdtrees(1)
    return s


TURN = np.array([[0.8, -0.6, 0], [0.6, 0.8, 0], [0, 0, 1]])


@pytest.mark.parametrize("make,wide", [
    (lambda: soup(1, 1), True), (lambda: soup(1025, 2), True), (lambda: soup(3000, 5, 1e-6), True),
    (lambda: soup(3000, 5, 1e6), True), (lambda: soup(3000, 5, 1.0, -30000.0), True),
    (lambda: soup(2000, 7, copies=900), True), (lambda: scenes.hard_lighting_room(cells=24), True),
    (lambda: FlatScene.read(golden("cornell_alpha_64.yfs")), True),
    (lambda: soup(3000, 5, 1e-12), False), (lambda: soup(3000, 5, 1e12), False),
    (lambda: moved(soup(3000, 5), TURN), False), (lambda: moved(soup(3000, 5), 1.5 * np.eye(3)), False)],
    ids=["one", "1025", "small", "large", "far", "copies", "walls", "alpha", "too small", "too large",
         "one of two rotated", "one of two scaled"])
def test_which_scenes_have_a_wide_tree(make, wide):
    """The scenes that the settling is tested on do cast through the tree, and
    those that it does not take walk the kd-tree, with its results."""
    s = make()
    assert casts_through_wide_tree(s) == wide
    assert_settled(s, probing_rays(s, 4096, 34))


def doubled(s, part):
    """The scene with the first `part` of every mesh's triangles once more, their
    vertices in another order."""
    for m in s.meshes:
        again = m.indices[:int(part * m.triangle_count)][:, [0, 2, 1]]
        m.indices = np.concatenate([m.indices, again])
    s.build_kdtrees(1)
    return s


@pytest.mark.parametrize("part,timed", [(0.0, False), (0.1, False), (0.3, True), (1.0, True)])
def test_scenes_of_twins(part, timed):
    """Where many triangles are there twice, closest hits (near ties) are timed
    among the kd-tree kernels; shadow rays keep the wide tree."""
    s = doubled(soup(3000, 41), part)
    ctx = native.Context(0)
    try:
        ctx.upload_scene(s)
        lo, hi = scenes.scene_box(s)
        rays = scenes.random_rays(lo, hi, TIMED_RAYS, 62)
        ctx.cast_closest(rays)
        ctx.cast_any(rays)
        kernels = ctx.traversal_kernels()["cast"]
    finally:
        ctx.close()
    assert (kernels[0] != 0) == timed and kernels[1] == 0
    assert_settled(s, probing_rays(s, 16384, 42))


def test_twins_of_a_render():
    s = FlatScene.read(golden("cornell_c1_64.yfs"))
    s.config["render_region"] = (0, 0, 256, 256)
    s.camera["image_extent"] = (256, 256)
    s = doubled(s, 1.0)
    got = []
    for kernel in (native.TRAVERSAL_AUTO, native.TRAVERSAL_PER_RAY):
        ctx = native.Context(0, traversal_kernel=kernel)
        try:
            ctx.upload_scene(s)
            got += [ctx.render(256, 256) for _ in range(2)]
            kernels = ctx.traversal_kernels()
            if kernel == native.TRAVERSAL_AUTO:
                assert kernels["render_closest"][0] != 0 and kernels["render_any"] == [0] * 5
        finally:
            ctx.close()
    for img, stats in got[1:]:
        assert img.tobytes() == got[0][0].tobytes() and stats.variance == got[0][1].variance


def test_object_placed_twice():
    """Twins of two objects with one mesh; a third place is no twin."""
    def place(*shifts):
        s = soup(1000, 43)
        s.meshes = s.meshes[1:]
        m = np.eye(3, 4, dtype=np.float32)
        objects = []
        for shift in shifts:
            m[:, 3] = shift
            w = np.eye(3, 4, dtype=np.float32)
            w[:, 3] = -m[:, 3]
            objects.append(make_object(0, m.ravel().copy(), w.ravel().copy()))
        s.objects = np.array(objects)
        s.build_kdtrees(1)
        return s
    for shifts, wide in (((0.5, 0.5), False), ((0.5, 2.5), True)):
        s = place(*shifts)
        ctx = native.Context(0)
        try:
            ctx.upload_scene(s)
            lo, hi = scenes.scene_box(s)
            ctx.cast_closest(scenes.random_rays(lo, hi, TIMED_RAYS, 63))
            assert (ctx.traversal_kernels()["cast"][0] == 0) == wide
        finally:
            ctx.close()
        assert_settled(s, probing_rays(s, 16384, 44))


def test_rays_from_far_away():
    """Rays from origins that the tree's margins do not cover walk the kd-tree;
    after a batch of them the casts are timed among the kd-tree kernels.  Small
    batches and nearer ones change nothing."""
    s = soup(5000, 51)
    lo, hi = scenes.scene_box(s)
    rays = scenes.random_rays(lo, hi, TIMED_RAYS, 64)
    far = rays.copy()
    far[:, 0:3] -= np.float32(1000) * far[:, 4:7]
    some = rays.copy()
    some[::6] = far[::6]
    want = native.Context(0, traversal_kernel=native.TRAVERSAL_PER_RAY)
    ctx = native.Context(0)
    try:
        for c in (ctx, want):
            c.upload_scene(s)
        for batch, n, kernels in ((rays, TIMED_RAYS, (True, True)), (some, TIMED_RAYS, (True, True)),
                                  (far, 60000, (True, True)), (far, TIMED_RAYS, (True, True)),
                                  (far, TIMED_RAYS, (False, True)), (rays, TIMED_RAYS, (False, True))):
            got, ref = ctx.cast_closest(batch[:n]), want.cast_closest(batch[:n])
            for g, w in zip(got, ref):
                assert g.tobytes() == w.tobytes()
            assert tuple(k == 0 for k in ctx.traversal_kernels()["cast"]) == kernels
        for batch in (far, far):
            assert ctx.cast_any(batch).tobytes() == want.cast_any(batch).tobytes()
        assert 0 not in ctx.traversal_kernels()["cast"]
        ctx.upload_scene(s)
        assert ctx.traversal_kernels()["cast"] == [0, 0]
        ctx.cast_closest(rays)
        assert ctx.traversal_kernels()["cast"] == [0, 0]
    finally:
        ctx.close()
        want.close()
