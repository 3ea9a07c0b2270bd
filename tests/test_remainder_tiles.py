"""When a batch's last strings run in a smaller tile (host side): a sweep of its own, so only
where the tables it saves are worth its launches."""
import ctypes

import numpy as np
import pytest


def _plan(pkg, rank, n):
    for s in range(4000):
        rng = np.random.default_rng(s)
        g = pkg.instances.degree_at_most3(n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if max(pkg.rank_profile(n, e, order)) == rank:
            return pkg.ScanPlan(n, e, order)
    raise AssertionError("no such plan")


def _launches(pkg, plan, batch, tile, precision):
    ws, out = ctypes.c_size_t(), ctypes.c_int64()
    prec = pkg.PRECISIONS[precision]
    pkg._lib.check(pkg._lib.lib().rgs_scan_workspace_bytes(plan.handle, tile, prec, ctypes.byref(ws)))
    pkg._lib.check(pkg._lib.lib().rgs_scan_launch_count(plan.handle, batch, tile, prec, ws, ctypes.byref(out)))
    return out.value


@pytest.mark.parametrize("rank,n,batch,tile,precision,split", [
    (13, 32, 5, 4, "c64", 0), (13, 32, 300, 128, "c64f32", 0), (15, 36, 33, 32, "c128", 0), (17, 40, 33, 32, "c64f32", 0),
    (17, 40, 65, 64, "c128", 0), (17, 40, 129, 128, "c64", 0), (17, 40, 257, 256, "c64f32", 1),
    (18, 44, 40, 32, "c64", 8), (19, 46, 3, 2, "c64f32", 0), (20, 46, 5, 4, "c64f32", 0), (20, 46, 70, 64, "c128", 8),
    (22, 50, 3, 2, "c128", 0), (22, 50, 11, 8, "c64f32", 4), (24, 56, 5, 4, "c64f32", 1)])
def test_remainder_rule(pkg, rank, n, batch, tile, precision, split):
    plan = _plan(pkg, rank, n)
    whole = -(-batch // tile) * tile  # as many full tiles
    count = _launches(pkg, plan, batch, tile, precision)
    if split:
        assert count == _launches(pkg, plan, batch - batch % tile, tile, precision) + \
            _launches(pkg, plan, batch % tile, split, precision)
    else:
        assert count == _launches(pkg, plan, whole, tile, precision)
