"""Routes that larger plans, smaller tiles or more strings take: the chain sampler on chip and
streamed against the statevector in every precision, several strings per warp in samples and
conditionals, the tuned tile of a streamed plan, and the step codes that runs meet.
"""
import numpy as np
import pytest

from oracle import graph_state as gs
from oracle import scan_plan as sp

pytestmark = pytest.mark.gpu

PRECISIONS = ["c64", "c64f32", "c128"]


def _plan(pkg, rank, n, seed=0):
    while True:
        seed += 1
        rng = np.random.default_rng(seed)
        g = [pkg.instances.degree_at_most3, pkg.instances.erdos_renyi][seed % 2](n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if max(pkg.rank_profile(n, e, order)) == rank:
            return g, pkg.instances.haar_su2(n, rng), order


@pytest.mark.parametrize("precision,tol", [("c64", 1e-5), ("c64f32", 1e-4), ("c128", 1e-10)])
@pytest.mark.parametrize("tile", [None, 16, 2])
@pytest.mark.parametrize("kind,n,seed", [("reg3", 12, 1), ("dense", 10, 2), ("er3", 14, 3), ("deg3", 16, 4)])
def test_chain_routes_match_oracle(pkg, kind, n, seed, tile, precision, tol):
    """Draws with given uniforms, conditionals, log p and p: the default tile runs on chip, the
    smaller ones the Gram, pair-Gram and decision kernels.  Bounds as for the sampler's own
    oracle test: 1e-5 of a branch boundary, the storage precision of conditionals and p."""
    inst = pkg.instances.make_instance(kind, n, seed, pkg.rank_profile)
    probs = np.abs(gs.statevector(inst.g, inst.u)) ** 2
    cs = pkg.ChainSampler(inst.g, inst.u, inst.order, precision=precision, batch_tile=tile)
    assert cs.plan.pairs and (cs.launch_count(100) == 1) == (tile is None)
    uni = np.random.default_rng(seed).random((100, n))
    bits, p, logp, cond = cs.sample(100, uniforms=uni, with_conditionals=True)
    matched = 0
    for i in range(100):
        ref, margins = gs.chain_sample(probs, inst.order, uni[i])
        if margins.min() < 1e-5:
            continue
        assert np.array_equal(bits[i], ref)
        idx = int((ref.astype(np.int64) << np.arange(n)).sum())
        assert abs(p[i] - probs[idx]) / probs[idx] < (1e-12 if precision == "c128" else 1e-4)
        assert abs(logp[i] - np.log(probs[idx])) < (1e-9 if precision == "c128" else 1e-4)
        matched += 1
    assert matched > 95
    given, lp, q = cs.marginals(bits)
    assert np.array_equal(p, q) and np.abs(given - cond).max() < 1e-6
    for i in range(0, 100, 9):
        assert np.abs(cond[i] - gs.chain_conditionals(probs, inst.order, bits[i])).max() < max(tol, 2e-7)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("rank,n,counts", [(3, 10, (1200, 9500, 19000)), (5, 14, (2400, 9501)), (7, 18, (1185, 2369)),
                                           (8, 20, (1300,)), (9, 22, (1300,))])
def test_strings_sharing_a_warp(pkg, rank, n, counts, precision):
    """Samples and conditionals of batches large enough for 2 to 32 strings per warp (partly
    filled last units) against position-by-position plans: draws and p equal, log p over sums
    of at most 2^9 float64 terms in another order to 1e-9, float32 conditionals to one rounding."""
    g, u, order = _plan(pkg, rank, n)
    e = pkg.edges_from_graph(g)
    on = pkg.ChainSampler(g, u, order, precision=precision, plan=pkg.ScanPlan(n, e, order))
    off = pkg.ChainSampler(g, u, order, precision=precision, plan=pkg.ScanPlan(n, e, order, fuse=False))
    for count in counts:
        assert on.launch_count(count) == 1 < off.launch_count(count)
        (xa, pa, qa, da), (xb, pb, qb, db) = (c.sample(count, seed=count, with_conditionals=True) for c in (on, off))
        assert np.array_equal(xa, xb) and np.array_equal(pa, pb)
        assert np.abs(qa - qb).max() < 1e-9 and np.abs(da - db).max() <= 2.0 ** -23
        (da, qa, pa), (db, qb, pb) = on.marginals(xa[::-1]), off.marginals(xa[::-1])
        assert np.array_equal(pa, pb)
        assert np.abs(qa - qb).max() < 1e-9 and np.abs(da - db).max() <= 2.0 ** -23


@pytest.mark.parametrize("precision", PRECISIONS)
def test_tuned_tile_of_a_streamed_plan(pkg, precision):
    """batch_tile='tune' where the tile matters (rank 13, fused pairs): the result is that of
    any tile, bitwise."""
    g, u, order = _plan(pkg, 13, 32)
    plan = pkg.ScanPlan(32, pkg.edges_from_graph(g), order)
    bits = pkg.instances.uniform_bits(300, 32, np.random.default_rng(3))
    tuned = pkg.ScanEngine(plan, u, precision=precision, batch_tile="tune")
    val, ls = tuned.sweep_bits(bits)
    best, rates = tuned.tuning
    assert plan.pairs and tuned.launch_count(300) > 1 and len(rates) > 3 and rates[best] == max(rates.values())
    for tile in (1, 8):
        v, l = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile).sweep_bits(bits)
        assert np.array_equal(val, v) and np.array_equal(ls, l)


def test_runs_meet_every_step_code(pkg):
    """The positions inside the runs of the plans that the bitwise route test sweeps have every
    step code there is: 1, 2 or 4 gathers to a pair of rows, with and without y bits among them,
    1 or 2 to one row.  (Four gathers without y bits cannot occur: a position consumes one bit.)"""
    from test_route_bits_gpu import _instances
    codes = set()
    for n, e, order, _ in _instances(pkg, 18, 19, 3, 10, (34, 44)):
        steps, _ = sp.make_plan(n, e, order)
        for j, k in pkg.ScanPlan(n, e, order).segments:
            for st in steps[j:j + k] if k > 2 else []:
                y, span = 1 << st.r_in, sp.kernel_combos(st.kernel)
                codes.add((y in span, len(span), any(c & y for c in span)))
    assert codes == {(False, 1, False), (False, 2, False), (False, 2, True), (False, 4, True), (True, 2, True),
                     (True, 4, True)}
