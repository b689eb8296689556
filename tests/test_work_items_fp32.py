"""The FP32-velocity variant's work items on basins whose strips hold runs of
land: within the variant's tolerances of the FP64 oracle after 10 steps, land
and halo points unchanged."""
import numpy as np
import pytest
from conftest import rel_err

from inmsom_elfs_b200.grid import STATE
from test_fp32_velocity import TOL_SSH, TOL_UV
from test_work_items import _banded

pytestmark = pytest.mark.gpu

CASES = [
    (31, 40, [(3, 1), (9, 7), (20, 8), (31, 5)]),
    (62, 60, [(2, 9), (13, 8), (23, 10), (40, 20)]),
    (400, 170, [(10, 9), (21, 8), (60, 30), (100, 1), (140, 12)]),
    (700, 500, [(1, 40), (60, 9), (200, 8), (300, 100)]),
    (1300, 1300, [(5, 9), (400, 8), (700, 200)]),
]


@pytest.mark.parametrize("nx,ny,bands", CASES)
def test_land_runs_with_fp32_velocities(gpu, ora, nx, ny, bands):
    b = _banded(ora, nx, ny, bands, seed=nx + ny)
    bo, bg = b.copy(), b.copy()
    with gpu.BarotropicSolver(bg, resident=True, fp32_velocity=True) as s:
        assert s.path()[0] == 1
        s.load_state()
        s.run_substeps(10, b.dt)
        s.sync_to_host()
    ora.run_substeps(bo, 10, b.dt)
    land = b.masks["lu"] < 0.5
    for k in STATE:
        assert rel_err(bg.state[k], bo.state[k]) <= (TOL_SSH if k.startswith("ssh") else TOL_UV), k
        assert np.array_equal(bg.state[k][land], b.state[k][land]), k
