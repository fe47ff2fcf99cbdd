"""What bench.py says of the cast kernels: the bytes of the calls that it
times, and the traffic of the kernels that they launch."""
import bench


def test_cast_roofline_is_of_the_kernels_it_times():
    triangles, rays = 2424832, 1 << 24
    r = bench.cast_roofline(triangles, rays, 4.26, 6777.2, "measured")
    compulsory = 52 * rays + 36 * triangles  # no node of a tree that the call does not walk
    assert abs(r["algorithmic_bytes_per_ray"] * rays - compulsory) < 0.1 * rays
    assert abs(r["frac"] - compulsory / 4.26e-3 / 6777.2e9) < 1e-4
    assert "cast_wide" in r["kernel"] and "settle_wide" in r["kernel"]
    assert compulsory < r["traffic"] < 6777.2e9 * 4.26e-3  # what the chip can move meanwhile
