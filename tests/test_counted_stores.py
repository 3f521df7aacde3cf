"""Stores into another block of a cluster that count themselves on its barrier (st.async) complete that barrier with release
at cluster scope.  A wait whose acquire reaches this block only does not order the loads of the stored values after them, and
no run shows it: so the sources are read, and each barrier that is counted on has to be waited for by mbar_wait_counted.  The
reference has no counterpart (its kernels launch no clusters)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aotx_b200", "csrc")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_every_counted_barrier_is_acquired_at_cluster_scope():
    users = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        code = _code(path)
        barriers = re.findall(r"store_counted\([^;]*,\s*mapa_shared\((\w+),[^;]*\);", code)
        assert len(barriers) == code.count("store_counted("), path
        for name in set(barriers):
            waits = re.findall(r"(mbar_\w*wait\w*)\(\s*%s\b" % name, code)
            assert waits and set(waits) == {"mbar_wait_counted"}, (path, name, waits)
            users += 1
    assert users >= 2
    assert ".acquire.cluster" in _code(os.path.join(CSRC, "q8_ptx.cuh"))
