"""The work items of ensemble members: about 16 rows, to the nearest, where the
members are small (a segment of 31 rows is two items, not one: with few
members the longest chain of rows sets the time), and the members' values are
those of the basins run alone, bit for bit."""
import ctypes

import numpy as np
import pytest

from inmsom_elfs_b200 import _lib, basins
from inmsom_elfs_b200.grid import STATE

pytestmark = pytest.mark.gpu


def _items(s, table=0):
    n, rows = ctypes.c_int(), ctypes.c_int()
    assert _lib.load().inmsom_test_items(s._ctx, table, ctypes.byref(n), ctypes.byref(rows)) == _lib.OK
    return n.value, rows.value


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("ny", [7, 15, 16, 23, 24, 31, 32, 39, 40, 63, 170])
def test_members_items_of_about_16_rows(gpu, ora, ny, persistent):
    b = basins.beta_plane_basin(n=70, ny=ny, seed=ny)
    basins.finalize(b, ora.OracleBackend())
    rng = np.random.default_rng(ny)
    for k in ("ssh_e", "sshp_e"):
        b.state[k] = np.asfortranarray(0.1 * rng.standard_normal(b.bounds.shape) * b.masks["lu"])
    alone, a, c = b.copy(), b.copy(), b.copy()
    with gpu.BarotropicSolver(alone, resident=True) as s:
        s.load_state()
        s.run_substeps(4, b.dt)
        s.sync_to_host()
    members = [gpu.BarotropicSolver(x, resident=True) for x in (a, c)]
    for s in members:
        s.load_state()
    with gpu.Ensemble(members, group=2, persistent=persistent) as e:
        assert _items(members[0])[1] <= 24
        e.run(4, [b.dt] * 2)
    for s, x in zip(members, (a, c)):
        s.sync_to_host()
        s.close()
        for k in STATE:
            assert np.array_equal(x.state[k], alone.state[k]), k


def test_items_argument_checks():
    n = ctypes.c_int()
    assert _lib.load().inmsom_test_items(None, 0, ctypes.byref(n), ctypes.byref(n)) == _lib.EARG
