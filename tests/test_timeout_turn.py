"""The bounded-wait hook on a table whose alternate substeps run through the
items from the other end: it withholds the rows of the same work item in
every substep, not of the item at the same place in the launch."""
import numpy as np
import pytest

from inmsom_elfs_b200 import _lib, basins

pytestmark = pytest.mark.gpu


def test_hold_names_an_item_in_every_substep(gpu, ora):
    b = basins.beta_plane_basin(n=1300, seed=3)     # some 60 000 rows: several waves of items
    basins.finalize(b, ora.OracleBackend())
    rng = np.random.default_rng(3)
    for k in ("ssh_e", "sshp_e"):
        b.state[k] = np.asfortranarray(0.1 * rng.standard_normal(b.bounds.shape) * b.masks["lu"])
    ora.hh_init_external(b)
    bg = b.copy()
    lib = _lib.load()
    with gpu.BarotropicSolver(bg, resident=True) as s:
        assert s.path()[0] == 1
        s.load_state()
        assert lib.inmsom_test_hold_copy(s._ctx, 0, 0, 4096) == _lib.OK
        assert lib.inmsom_run_substeps(s._ctx, 2, b.dt, None, None) == _lib.ETIMEOUT
        assert lib.inmsom_test_hold_copy(s._ctx, -1, 0, 0) == _lib.OK
        s.sync_to_host()
    wet = np.argwhere(b.masks["lu"].T > 0.5)        # (row, column), row by row
    south, north = wet[wet[:, 0] == wet[0, 0]], wet[wet[:, 0] == wet[-1, 0]]
    # item 0: the southernmost rows of the first strip; the last item: the
    # northernmost rows of the last strip
    first, last = (south[0][1], south[0][0]), (north[-1][1], north[-1][0])
    assert bg.state["ssh_e"][first] == b.state["ssh_e"][first]
    assert bg.state["ssh_e"][last] != b.state["ssh_e"][last]
