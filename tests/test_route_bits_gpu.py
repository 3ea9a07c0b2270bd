"""A string's (value, logscale) has the same bits whatever call it is part of: any count of
strings (plans of rank <= 12 are swept on chip, in fused pairs or in runs by the count), any
tile, with or without fusion, in an amplitude call, a chain-sampler call or a resident batch.

Every schedule sums the same terms of an entry in the same order and rounds it to the
storage type, so tables agree up to powers of two; the last position runs alone, scaled
from the true maximum of the table before it, which fixes the sum of the exponents.
Equality is exact (no entry of these instances is near the underflow of its type).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRECISIONS = ["c64", "c64f32", "c128"]


def _instances(pkg, low, high, count, seed, sizes):
    rng = np.random.default_rng(seed)
    out, k = [], 0
    while len(out) < count:
        k += 1
        n = 2 * int(rng.integers(sizes[0] // 2, sizes[1] // 2 + 1))
        make = [pkg.instances.regular3, pkg.instances.erdos_renyi, pkg.instances.degree_at_most3,
                pkg.instances.dense][k % 4]
        if make is pkg.instances.dense and n > 2 * high - 2:
            continue
        g = make(n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if low <= max(pkg.rank_profile(n, e, order)) <= high:
            out.append((n, e, order, pkg.instances.haar_su2(n, rng)))
    return out


def _same(a, b, what):
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), what


def _check_counts(pkg, n, e, order, u, precision, many, rng):
    """Fused calls of every size against one unfused call."""
    single = pkg.ScanEngine(pkg.ScanPlan(n, e, order, fuse=False), u, precision=precision, batch_tile=32)
    bits = pkg.instances.uniform_bits(many, n, rng)
    val, ls = single.sweep_bits(bits)
    plan = pkg.ScanPlan(n, e, order)
    launches = set()
    for tile in (8, pkg.max_batch_tile(precision)):
        eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
        for count in sorted({1, 32, 33, 100, 127, 128, 700, many}):
            if count <= many:
                launches.add(eng.launch_count(count))
                _same(eng.sweep_bits(bits[:count]), (val[:count], ls[:count]), (plan.rmax, tile, count))
    return plan, launches


@pytest.mark.parametrize("precision", PRECISIONS)
def test_counts_of_low_rank_plans(pkg, precision):
    from test_pair_fusion import rare_code_plans
    rng = np.random.default_rng(1)
    cases = _instances(pkg, 3, 12, 10, 5, (10, 30))
    for g, order in rare_code_plans(pkg).values():
        cases.append((len(g), pkg.edges_from_graph(g), order, pkg.instances.haar_su2(len(g), rng)))
    codes = set()
    for n, e, order, u in cases:
        plan, launches = _check_counts(pkg, n, e, order, u, precision, 700, rng)
        assert 1 in launches and max(launches) > 1
        codes |= {(plan.pair_info(k).code_a, plan.pair_info(k).code_b) for k in range(len(plan.pairs))}
    assert len(codes) >= 15 and {c for p in codes for c in p} == {0, 1, 2, 3, 4}, codes


@pytest.mark.parametrize("precision,rank", [("c64", 12), ("c64", 10), ("c64f32", 12), ("c64f32", 11), ("c128", 12),
                                            ("c128", 10)])
def test_runs_over_all_positions(pkg, precision, rank):
    """Batches from which these plans run as runs: 2^23 complex64 entries, or 512 strings."""
    rng = np.random.default_rng(rank)
    many = 600 if (precision, rank) == ("c128", 12) else (1 << (23 - rank)) + 5
    for n, e, order, u in _instances(pkg, rank, rank, 3, 40 + rank, (22, 34)):
        plan, launches = _check_counts(pkg, n, e, order, u, precision, many, rng)
        assert 1 in launches and pkg.ScanEngine(plan, u, precision=precision).launch_count(many) > 1


@pytest.mark.parametrize("precision", PRECISIONS)
def test_tiles_of_streamed_plans(pkg, precision):
    """Ranks 13 to 16 (fused pairs) and 18 to 19 (runs), every tile, against single positions."""
    rng = np.random.default_rng(3)
    for n, e, order, u in _instances(pkg, 13, 16, 4, 9, (26, 40)) + _instances(pkg, 18, 19, 3, 10, (34, 44)):
        plan, single = pkg.ScanPlan(n, e, order), pkg.ScanPlan(n, e, order, fuse=False)
        bits = pkg.instances.uniform_bits(70, n, rng)
        ref = pkg.ScanEngine(single, u, precision=precision, batch_tile=8).sweep_bits(bits)
        for tile in (1, 2, 16, 64, pkg.max_batch_tile(precision)):
            eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
            assert eng.launch_count(70) > 1
            _same(eng.sweep_bits(bits), ref, (plan.rmax, tile))
            _same(eng.sweep_bits(bits[:11]), (ref[0][:11], ref[1][:11]), (plan.rmax, tile))


@pytest.mark.parametrize("precision", PRECISIONS)
def test_chain_and_batch(pkg, precision):
    """p(x) of the chain sampler on chip, streamed in tiles and unfused, and the amplitudes of
    a resident batch."""
    rng = np.random.default_rng(4)
    for n, e, order, u in _instances(pkg, 6, 12, 3, 21, (16, 30)) + _instances(pkg, 13, 14, 1, 22, (28, 34)):
        g = np.zeros((n, n), dtype=np.uint8)
        for a, b in e:
            g[a, b] = g[b, a] = 1
        plan, single = pkg.ScanPlan(n, e, order), pkg.ScanPlan(n, e, order, fuse=False)
        bits = pkg.instances.uniform_bits(150, n, rng)
        ref = pkg.ScanEngine(single, u, precision=precision).sweep_bits(bits)
        p = np.abs(pkg.amplitudes_from(*ref, n)) ** 2
        for pl, tile in ((plan, None), (plan, 16), (single, 32)):
            _, _, q = pkg.ChainSampler(g, u, order, precision=precision, plan=pl, batch_tile=tile).marginals(bits)
            assert np.array_equal(p, q), (plan.rmax, tile)
        if plan.rmax <= 12:
            rb = pkg.ResidentBatch(precision)
            k = rb.add(g, u, order, bits)
            rb.run()
            _same(rb.amplitudes(k)[:2], ref, plan.rmax)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("rank", [21, 23])
def test_single_strings(pkg, precision, rank):
    """One string per tile, where complex64 plans of some ranks keep their pairs instead of
    runs, and remainder tiles of one, against single positions."""
    rng = np.random.default_rng(rank)
    for n, e, order, u in _instances(pkg, rank, rank, 1, 60 + rank, (44, 52)):
        bits = pkg.instances.uniform_bits(5, n, rng)
        ref = pkg.ScanEngine(pkg.ScanPlan(n, e, order, fuse=False), u, precision=precision, batch_tile=2).sweep_bits(bits)
        plan = pkg.ScanPlan(n, e, order)
        counts = {}
        for tile in (1, 4):
            eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
            counts[tile] = eng.launch_count(tile)
            _same(eng.sweep_bits(bits), ref, (rank, tile))
        pairs = precision == "c64f32" or (precision == "c64" and rank == 21)
        assert (counts[1] > counts[4]) == pairs
