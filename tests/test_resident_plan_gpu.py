"""Low-rank plans on chip (one launch, tables in shared memory) against the streamed
executors, which plans without fused pairs (``fuse=False``) still use.

The on-chip sweep does the position-by-position arithmetic in the same order, so values
and log-scales are bitwise equal.  Branch masses are float64 sums in another order: log p
over n <= 60 positions of sums of at most 2^12 terms agrees to 1e-9, conditionals are the
same float32 up to one rounding (2^-23 relative, 2^-24 absolute at 1), and a draw can only
differ where its uniform lies within that of a branch boundary (never, for these seeds,
unless a sum is wrong).  Ranks cover one and several strings per warp, one and four warps
per unit, and both table sizes; counts cover partly filled units and both ends of the
batch sizes the scan takes on chip.  Also here: the fused pair kernel at every pair code,
on batches that stay streamed.
"""
import numpy as np
import pytest

from oracle import graph_state as gs

pytestmark = pytest.mark.gpu


def _plans(pkg, rank):
    """A seeded degree-<=3 instance whose searched or random order has this max rank."""
    for s in range(2000):
        rng = np.random.default_rng(s)
        n = {3: 12, 6: 20, 8: 24, 9: 40, 10: 26, 11: 28, 12: 30}[rank]
        g = pkg.instances.degree_at_most3(n, rng)
        order = rng.permutation(n).tolist()
        if rank <= 9:
            order, _, _ = pkg.search_order(n, pkg.edges_from_graph(g), order, iterations=500, seed=1, threads=1)
        if max(pkg.rank_profile(n, pkg.edges_from_graph(g), order)) == rank:
            u = pkg.instances.haar_su2(n, rng)
            e = pkg.edges_from_graph(g)
            return g, u, order, pkg.ScanPlan(n, e, order), pkg.ScanPlan(n, e, order, fuse=False)
    raise AssertionError("no such instance")


@pytest.mark.parametrize("precision", ["c64", "c64f32", "c128"])
@pytest.mark.parametrize("rank", [3, 6, 8, 9, 10, 11, 12])
def test_on_chip_equals_streamed(pkg, rank, precision):
    g, u, order, plan, streamed = _plans(pkg, rank)
    n = len(g)
    rng = np.random.default_rng(rank)
    a = pkg.ScanEngine(plan, u, precision=precision)
    b = pkg.ScanEngine(streamed, u, precision=precision)
    for count in (1, 32, 128, 1300):
        assert a.launch_count(count) == 1 or (precision == "c128" and rank >= 12 and count >= 512)
        bits = pkg.instances.uniform_bits(count, n, rng)
        (va, la), (vb, lb) = a.sweep_bits(bits), b.sweep_bits(bits)
        if a.launch_count(count) == 1:
            assert np.array_equal(va, vb) and np.array_equal(la, lb), (rank, count)
    fvec = rng.normal(size=(7, n, 2)) + 1j * rng.normal(size=(7, n, 2))
    (va, la), (vb, lb) = a.sweep_fvec(fvec), b.sweep_fvec(fvec)
    assert np.array_equal(va, vb) and np.array_equal(la, lb)

    ca = pkg.ChainSampler(g, u, order, precision=precision, plan=plan)
    cb = pkg.ChainSampler(g, u, order, precision=precision, plan=streamed)
    for count in (1, 75, 700):
        assert ca.launch_count(count) == 1 < cb.launch_count(count)
        uni = rng.random((count, n))
        for kw in (dict(uniforms=uni), dict(seed=11 + count)):
            (xa, pa, qa, da), (xb, pb, qb, db) = (c.sample(count, with_conditionals=True, **kw) for c in (ca, cb))
            assert np.array_equal(xa, xb) and np.array_equal(pa, pb)
            assert np.abs(qa - qb).max() < 1e-9
            assert np.abs(da - db).max() <= 2.0 ** -23
        (da, qa, pa), (db, qb, pb) = ca.marginals(xa), cb.marginals(xa)
        assert np.array_equal(pa, pb) and np.abs(qa - qb).max() < 1e-9 and np.abs(da - db).max() <= 2.0 ** -23


def test_small_tiles_and_zero_probability(pkg):
    """A tile below 64 keeps the streamed schedule, with the same draws; marginals of strings
    of probability 0 keep p = 0 and a log p of rounding size (below -30), as streamed."""
    g, u, order, plan, streamed = _plans(pkg, 6)
    whole = pkg.ChainSampler(g, u, order, plan=plan).sample(100, seed=5, with_conditionals=True)
    tiles = pkg.ChainSampler(g, u, order, plan=plan, batch_tile=16)
    assert tiles.launch_count(100) == 7 * tiles.launch_count(16) > 7
    bits, p, logp, cond = tiles.sample(100, seed=5, with_conditionals=True)
    assert np.array_equal(bits, whole[0]) and np.allclose(p, whole[1], rtol=1e-5, atol=0)
    assert np.abs(logp - whole[2]).max() < 1e-4 and np.abs(cond - whole[3]).max() < 1e-4
    product = np.zeros((4, 4), dtype=np.uint8)           # edge-free graph, identity gates: |+>^4
    eye = np.tile(np.array([[1, 1], [1, -1]]) / np.sqrt(2), (4, 1, 1)).astype(np.complex128)
    strings = np.array([[0, 0, 0, 0], [0, 1, 0, 0]], dtype=np.uint8)
    for fuse in (True, False):
        c = pkg.ChainSampler(product, eye, [2, 0, 3, 1],
                             plan=pkg.ScanPlan(4, [], [2, 0, 3, 1], fuse=fuse), precision="c128")
        cond, lp, p = c.marginals(strings)
        assert abs(p[0] - 1) < 1e-12 and p[1] == 0 and abs(lp[0]) < 1e-12 and lp[1] < -30


@pytest.mark.parametrize("precision,tol", [("c64", 1e-4), ("c64f32", 1e-4), ("c128", 1e-12)])
def test_pair_codes_on_streamed_batches(pkg, precision, tol):
    """The pair kernel at every code the graphs and the rare-code plans give, on 100 strings
    (a batch that is streamed), at tiles 1, 16 and the largest, against the statevector."""
    from test_pair_fusion import rare_code_plans
    rng = np.random.default_rng(4)
    cases = list(rare_code_plans(pkg).values())
    for kind, n in (("reg3", 18), ("er3", 17), ("deg3", 18), ("dense", 13)):
        for _ in range(3):
            g = {"reg3": pkg.instances.regular3, "er3": pkg.instances.erdos_renyi,
                 "deg3": pkg.instances.degree_at_most3, "dense": pkg.instances.dense}[kind](n, rng)
            cases.append((g, rng.permutation(n).tolist()))
    for g, order in cases:
        n = len(g)
        u = pkg.instances.haar_su2(n, rng)
        plan = pkg.ScanPlan(n, pkg.edges_from_graph(g), order)
        bits = pkg.instances.uniform_bits(100, n, rng)
        ref = np.abs(gs.statevector(g, u)[(bits.astype(np.int64) << np.arange(n)).sum(axis=1)]) ** 2
        for tile in (1, 16, pkg.max_batch_tile(precision)):
            eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
            assert eng.launch_count(100) > 1
            p = np.abs(pkg.amplitudes_from(*eng.sweep_bits(bits), n)) ** 2
            assert np.max(np.abs(p - ref) / ref) < tol, (n, tile)
