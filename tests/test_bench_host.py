"""What bench.py says of the tensor work that its contractions execute, against a count of their tiles."""
import pytest

import bench


@pytest.mark.parametrize("n_ao", [1, 64, 65, 128, 129, 256, 400, 512])
def test_tensor_products_count_the_tiles(n_ao):
    mt, nt = -(-n_ao // 128), -(-n_ao // 64)
    # Mixed V_xc: 128 x 128 tiles; from two on the d_j planes are formed on and above the diagonal.
    tiles = [(a, b) for a in range(mt) for b in range(mt)]
    kinetic = [t for t in tiles if mt == 1 or t[0] <= t[1]]
    assert bench._tensor_products("vxc", "tf32x3", n_ao) == pytest.approx(
        6 * (len(tiles) + 3 * len(kinetic)) / (4 * len(tiles)))
    assert bench._tensor_products("density", "tf32x3", n_ao) == 3
    # FP64 V_xc: tiles of 128 x 64 that reach the diagonal; density: blocks of 64 up to it.
    tiles = [(a, b) for a in range(mt) for b in range(nt)]
    kinetic = [(a, b) for a, b in tiles if 64 * b + 63 >= 128 * a]
    assert bench._tensor_products("vxc", "fp64", n_ao) == pytest.approx(
        28 * (len(tiles) + 3 * len(kinetic)) / (4 * len(tiles)))
    assert bench._tensor_products("density", "fp64", n_ao) == pytest.approx(
        28 * (nt * nt + 3 * nt * (nt + 1) / 2) / (4 * nt * nt))
