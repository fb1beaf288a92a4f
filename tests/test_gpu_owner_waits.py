"""The give-up path of the sweeps whose rows are kept by their blocks: a row of
the block's own that nothing publishes, waited for as one of the four entries
that a row keeps at hand or as a further one; the wait record names both rows
by their places in the vectors."""
import ctypes as C
import re

import pytest

from blood_network_b200 import amg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, entries, limit_ms", [(2, 1, 5.0), (33, 1, 20.0), (22000, 1, 50.0),
                                                  (6, 5, 5.0), (256, 5, 20.0)])
def test_stalled_owner_sweep_names_the_rows(n, entries, limit_ms):
    lib = amg.load_library()
    ms = C.c_double(-1.0)
    rc = lib.amg_debug_wait_timeout_own(n, entries, limit_ms, C.byref(ms))
    msg = lib.amg_solver_last_error().decode()
    assert rc == amg.ERR_SPIN, (rc, msg)
    m = re.search(r"row (-?\d+) waited [0-9.]+ ms for row (-?\d+)", msg)
    assert m, msg
    row, dep = int(m.group(1)), int(m.group(2))
    # vectors in reverse: row r of the factor is n-1-r; the first row past the
    # independent ones waits for row 0, the others for the row before
    assert 0 <= row <= n - 1 - entries, msg
    assert dep == (n - 1 if row == n - 1 - entries else row + 1), msg
    # one limit for the launch; the chain then ends at a microsecond or so a row
    assert limit_ms * 0.9 <= ms.value <= limit_ms + 250.0, (ms.value, msg)


def test_owner_wait_selftest_rejects_bad_arguments():
    lib = amg.load_library()
    for args in ((1, 1, 10.0), (22001, 1, 10.0), (5, 5, 10.0), (257, 5, 10.0), (100, 2, 10.0),
                 (100, 1, 0.0), (100, 1, 1e6)):
        assert lib.amg_debug_wait_timeout_own(*args, None) == amg.ERR_ARG
