"""The benchmark's roofline counts ocean cells only: the substep skips runs of
land rows, so that bytes counted over every cell were never moved (0.97 of the
copy bandwidth on a basin with 40 % land)."""
import bench
from inmsom_elfs_b200 import basins


def test_algorithmic_bytes_are_those_of_ocean_cells(ora):
    b = basins.regional_basin(nx=61, ny=47, seed=4)
    basins.finalize(b, ora.OracleBackend())
    k = b.bounds
    ocean = sum(b.masks["lu"][m - k.bnd_x1, n - k.bnd_y1] > 0.5
                for m in range(k.nx_start, k.nx_end + 1) for n in range(k.ny_start, k.ny_end + 1))
    assert 0 < ocean < b.cells
    assert bench.substep_bytes(b, False) == 120 * ocean
    assert bench.substep_bytes(b, True) == 80 * ocean
