"""The wide tree answers a cast and the kd-tree settles it (csrc/wide_bvh.cuh):
every result is compared, bit for bit, with the kd-tree walked by one ray per
thread (the fixed traversal kernel), over triangle counts at the edges of the
builder, rays through vertices and edges, rays whose numbers the wide tree does
not cover, coincident triangles, trees that leave triangles out, meshes that
cast no shadow, and scenes far from or close to the origin."""
import numpy as np
import pytest

from conftest import cuda_available, golden
from yar_gb300 import native, scenes
from yar_gb300.scene import FlatScene, Mesh, make_object

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def soup(n, seed, scale=1.0, offset=0.0, copies=0):
    """n random triangles in the unit box (`copies` of them twice), two thirds of
    them in a second, translated object, one third axis-parallel."""
    rng = np.random.default_rng(seed)
    p = rng.random((n, 1, 3)) + 0.2 * (rng.random((n, 3, 3)) - 0.5)
    for a in range(3):
        k = np.arange(n) % 9 == a
        p[k, :, a] = p[k, :1, a]
    if copies:
        p[n - copies:] = p[:copies]
    p = (scale * (p + offset)).astype(np.float32)
    s = FlatScene()
    objects = []
    cut = n // 3
    for part, shift in ((p[:cut], 0.0), (p[cut:], 0.25 * scale)):
        if len(part) == 0:
            continue
        s.meshes.append(Mesh(part.reshape(-1, 3), np.arange(3 * len(part)).reshape(-1, 3)))
        m = np.array([1, 0, 0, shift, 0, 1, 0, -shift, 0, 0, 1, shift], np.float32)
        w = np.array([1, 0, 0, -shift, 0, 1, 0, shift, 0, 0, 1, -shift], np.float32)
        objects.append(make_object(len(s.meshes) - 1, m, w))
    s.objects = np.array(objects)
    s.build_kdtrees(1)
    return s


def probing_rays(s, n, seed):
    """Random rays, rays through vertices and edge points, axis-parallel rays, rays
    from far away, and rays with components that no margin covers."""
    rng = np.random.default_rng(seed)
    lo, hi = scenes.scene_box(s)
    size = hi - lo + 1e-3 * np.abs(hi).max()
    rays = scenes.random_rays(lo - 0.2 * size, hi + 0.2 * size, n, seed + 1, tmax=np.inf)
    q = n // 8
    m = s.meshes[-1]
    shift = np.asarray(s.objects[-1]["object_to_world"]).reshape(3, 4)[:, 3]
    tri = m.vertices[m.indices[rng.integers(0, m.triangle_count, 2 * q)]] + shift
    target = tri[:, 0].copy()
    target[q:] = 0.5 * (tri[q:, 0] + tri[q:, 1])
    rays[:2 * q, 4:7] = target - rays[:2 * q, 0:3]
    axis = rng.integers(0, 3, q)
    rays[2 * q:3 * q, 4:7] = 0.0
    rays[np.arange(2 * q, 3 * q), 4 + axis] = np.where(rng.random(q) < 0.5, -1, 1)
    rays[2 * q:3 * q, 0:3][np.arange(q), (axis + 1) % 3] = tri[:q, 1][np.arange(q), (axis + 1) % 3]
    rays[3 * q:4 * q, 0:3] += 50 * size * rays[3 * q:4 * q, 4:7]
    rays[3 * q:4 * q, 4:7] *= -1
    rays[4 * q:5 * q, 3] = rng.random(q) * np.linalg.norm(size)
    odd = rays[5 * q:5 * q + 64]
    odd[:8, 4] = 1e-12
    odd[8:16, 4:7] *= 1e-20
    odd[16:24, 5] = np.inf
    odd[24:32, 0] = np.nan
    odd[32:40, 3] = np.nan
    odd[40:48, 0:3] += 1e9
    odd[48:56, 4:7] = 0.0
    odd[56:64, 3] = -1.0
    return rays


def assert_settled(s, rays):
    if not cuda_available():
        pytest.skip("no CUDA device")
    got, want = [], []
    for out, kernel in ((got, native.TRAVERSAL_AUTO), (want, native.TRAVERSAL_PER_RAY)):
        ctx = native.Context(0, traversal_kernel=kernel)
        try:
            ctx.upload_scene(s)
            out += list(ctx.cast_closest(rays)) + [ctx.cast_any(rays)]
        finally:
            ctx.close()
    for k, name in ((1, "triangle"), (2, "object"), (4, "occlusion")):
        assert np.array_equal(got[k], want[k]), (name, np.nonzero(got[k] != want[k])[0][:8])
    assert np.array_equal(bits(got[0]), bits(want[0])) and np.array_equal(bits(got[3]), bits(want[3]))
    return got


@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 17, 65, 1023, 1024, 1025, 1027, 2049, 20000])
def test_triangle_counts(n):
    s = soup(n, n)
    got = assert_settled(s, probing_rays(s, 16384, n))
    assert (got[1] != 0xffffffff).any()


@pytest.mark.parametrize("scale,offset", [(1e-6, 0.0), (1e6, 0.0), (1.0, 1000.0), (1.0, -30000.0), (1e-12, 0.0), (1e12, 0.0)])
def test_scales_and_offsets(scale, offset):
    s = soup(3000, 5, scale, offset)
    assert_settled(s, probing_rays(s, 16384, 6))


def test_coincident_triangles():
    s = soup(2000, 7, copies=900)
    assert_settled(s, probing_rays(s, 32768, 8))


@pytest.mark.parametrize("which", ["leaf", "all"])
def test_trees_that_leave_triangles_out(which):
    """The tree decides what can be hit, not the mesh: leaves without their
    triangles (every third one, then every one)."""
    s = soup(4000, 9)
    for m in s.meshes:
        nodes = m.nodes.copy()
        todo, leaves = [0], []
        while todo:
            i = todo.pop()
            if nodes[i, 0] & 3 == 3:
                leaves.append(i)
            else:
                todo += [i + 1, int(nodes[i, 0] >> 2)]
        for i in leaves[::1 if which == "all" else 3]:
            nodes[i, 0] = 3
        m.nodes = nodes
    got = assert_settled(s, probing_rays(s, 16384, 10))
    assert (got[1] != 0xffffffff).any() == (which == "leaf")


def test_flat_walls_and_rays_that_leave_them():
    """Tessellated axis-parallel planes: rays that start a few units in the last
    place off a wall, on it, and inside the room."""
    s = scenes.hard_lighting_room(cells=24)
    rng = np.random.default_rng(3)
    rays = probing_rays(s, 65536, 11)
    axis, side = rng.integers(0, 3, 40000), rng.integers(0, 2, 40000)
    start = rng.uniform((-1, 0, -1), (1, 2, 1), (40000, 3)).astype(np.float32)
    wall = np.array([[-1, 1], [0, 2], [-1, 1]], np.float32)[axis, side]
    off = np.float32(1) * rng.integers(-300, 300, 40000).astype(np.float32) * np.float32(2.0 ** -23)
    start[np.arange(40000), axis] = wall + off
    rays[:40000, 0:3] = start
    rays[:40000, 4:7][np.arange(0, 40000, 2), axis[::2]] *= np.float32(1e-3)  # grazing
    assert_settled(s, rays)


@pytest.mark.parametrize("visibility", [1, 2])
def test_meshes_without_shadows(visibility):
    s = soup(3000, 12)
    s.meshes[0].visibility = visibility
    assert_settled(s, probing_rays(s, 16384, 13))


def test_alpha_tested_scene():
    s = FlatScene.read(golden("cornell_alpha_64.yfs"))
    assert_settled(s, probing_rays(s, 65536, 14))


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 200001])
def test_ray_counts(n):
    s = soup(5000, 15)
    assert_settled(s, probing_rays(s, max(n, 1024), 16)[:n])
