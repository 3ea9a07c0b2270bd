"""Passes of a streamed sweep (host side): they partition the positions in order, runs
appear from rank 18 on, and never cost more table entries than fused pairs alone."""
import numpy as np
import pytest


@pytest.mark.parametrize("kind,n,seed", [("regular3", 12, 1), ("regular3", 40, 2), ("degree_at_most3", 56, 3),
                                         ("erdos_renyi", 44, 4), ("regular3", 60, 5)])
def test_segments_partition(pkg, kind, n, seed):
    rng = np.random.default_rng(seed)
    g = getattr(pkg.instances, kind)(n, rng)
    for _ in range(4):
        order = rng.permutation(n).tolist()
        plan = pkg.ScanPlan(n, pkg.edges_from_graph(g), order)
        seg = plan.segments
        assert [j for j, _ in seg] == list(np.cumsum([0] + [k for _, k in seg])[:-1]) and sum(k for _, k in seg) == n
        if plan.rmax < 18:
            assert [j for j, k in seg if k == 2] == plan.pairs and max(k for _, k in seg) <= 2
        else:
            assert max(k for _, k in seg) > 2
        r = [0] + plan.ranks
        cost = sum(2 ** r[j] + 2 ** r[j + k] for j, k in seg)
        pairs = set(plan.pairs)
        one, j = 0, 0
        while j < n:
            k = 2 if j in pairs else 1
            one += 2 ** r[j] + 2 ** r[j + k]
            j += k
        assert cost <= one + 4096 * n
        off = pkg.ScanPlan(n, pkg.edges_from_graph(g), order, fuse=False)
        assert off.segments == [(j, 1) for j in range(n)]
