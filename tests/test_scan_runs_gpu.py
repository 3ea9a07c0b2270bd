"""Runs of positions (one pass, interior tables in shared memory) against the
position-by-position sweep, and remainder tiles.

Plans of rank 18 to 20 whose runs cover every step code the generator gives.  Both sweeps
round every entry to the storage type and differ in the power-of-two scales and in fused
multiply-add order nowhere, so amplitudes agree to the storage rounding of renormalised
tables: the repository's tolerances for fused against unfused sweeps (1e-4 float32
arithmetic, 1e-5 complex64, 1e-13 complex128 times n positions).  Tile results are bitwise
equal.  Contraction vectors of size 1e-9 and 1e9 run through the interior scales.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"c64": 1e-5, "c64f32": 1e-4, "c128": 1e-11}


def _plans(pkg, count, seed):
    rng = np.random.default_rng(seed)
    out, s = [], 0
    while len(out) < count:
        s += 1
        n = 2 * int(rng.integers(17, 28))
        g = [pkg.instances.regular3, pkg.instances.erdos_renyi, pkg.instances.degree_at_most3][s % 3](n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if 18 <= max(pkg.rank_profile(n, e, order)) <= 20:
            out.append((n, pkg.instances.haar_su2(n, rng), pkg.ScanPlan(n, e, order),
                        pkg.ScanPlan(n, e, order, fuse=False)))
    return out


@pytest.mark.parametrize("precision", ["c64", "c64f32", "c128"])
def test_runs_match_position_by_position(pkg, precision):
    import torch
    rng = np.random.default_rng(2)
    for n, u, plan, single in _plans(pkg, 4, 11):
        assert max(k for _, k in plan.segments) > 2 and all(k == 1 for _, k in single.segments)
        bits = pkg.instances.uniform_bits(24, n, rng)
        fvec = rng.normal(size=(24, n, 2)) + 1j * rng.normal(size=(24, n, 2))
        fvec *= 10.0 ** rng.choice([-9, 0, 0, 9], size=(24, n, 1))
        ref = pkg.ScanEngine(single, u, precision=precision, batch_tile=8)
        rv, rl = ref.sweep_bits(bits)
        fv, fl = ref.sweep_fvec(fvec)
        del ref
        outs = []
        for tile in (1, 2, 8, pkg.max_batch_tile(precision)):
            eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
            v, l = eng.sweep_bits(bits)
            amp, refamp = v * np.exp(l - 0.35 * n), rv * np.exp(rl - 0.35 * n)
            assert np.max(np.abs(np.abs(amp / refamp) ** 2 - 1)) < TOL[precision], tile
            w, m = eng.sweep_fvec(fvec)
            assert np.max(np.abs(np.abs(w / fv) ** 2 * np.exp(2 * (m - fl)) - 1)) < TOL[precision], tile
            outs.append((v, l, w, m))
            del eng
        for o in outs[1:]:
            assert all(np.array_equal(x, y) for x, y in zip(o, outs[0]))
        torch.cuda.empty_cache()


@pytest.mark.parametrize("precision,rank,count", [("c64f32", 12, 2050), ("c64", 11, 4099), ("c64f32", 10, 8192),
                                                  ("c128", 9, 8200), ("c128", 12, 513)])
def test_runs_over_all_positions(pkg, precision, rank, count):
    """Low-rank plans on batches large enough for runs over every position, at two tiles and
    with a workspace of one tile (bitwise equal), against complex128 position by position.
    Each of the n positions rounds an entry (arithmetic of up to four terms, then storage)
    by at most 4 units in the last place of the table's largest entries, and the sweep
    preserves norms, so an amplitude errs by at most n 2^-22 (complex64) or n 2^-50
    (complex128) of the largest one; small amplitudes have no relative bound of their own."""
    import torch
    for s in range(2000):
        rng = np.random.default_rng(s)
        n = {9: 22, 10: 24, 11: 26, 12: 30}[rank]
        g = pkg.instances.degree_at_most3(n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if max(pkg.rank_profile(n, e, order)) == rank:
            break
    u = pkg.instances.haar_su2(n, rng)
    plan, single = pkg.ScanPlan(n, e, order), pkg.ScanPlan(n, e, order, fuse=False)
    bits = pkg.instances.uniform_bits(count, n, rng)
    rv, rl = pkg.ScanEngine(single, u, precision="c128").sweep_bits(bits)
    ref = rv * np.exp(rl - 0.35 * n)
    eng = pkg.ScanEngine(plan, u, precision=precision)
    v, l = eng.sweep_bits(bits)
    assert 2 < eng.launch_count(count) < pkg.ScanEngine(single, u, precision=precision).launch_count(count)
    bound = n * 2.0 ** (-50 if precision == "c128" else -22) * np.abs(ref).max()
    assert np.abs(v * np.exp(l - 0.35 * n) - ref).max() <= bound
    small = pkg.ScanEngine(plan, u, precision=precision, batch_tile=16)
    w, m = small.sweep_bits(bits)
    assert np.array_equal(v, w) and np.array_equal(l, m)
    up = lambda x: (x + 255) // 256 * 256  # noqa: E731
    need = 2 * up((16 << rank) * small.esize) + up(n * 16 * 32) + up(n * 16) + up(n * 16 * 8)
    small._ws = torch.empty(need, dtype=torch.uint8, device=small.device)
    small.workspace_bytes = lambda tile: need
    w, m = small.sweep_bits(bits)
    assert np.array_equal(v, w) and np.array_equal(l, m)


def test_remainder_tile(pkg):
    """A batch's last strings run in the smallest tile that holds them: same results, and the
    launches that the launch count says."""
    n, u, plan, _ = _plans(pkg, 1, 5)[0]
    bits = pkg.instances.uniform_bits(11, n, np.random.default_rng(1))
    a = pkg.ScanEngine(plan, u, precision="c64f32", batch_tile=8)
    b = pkg.ScanEngine(plan, u, precision="c64f32", batch_tile=1)
    (va, la), (vb, lb) = a.sweep_bits(bits), b.sweep_bits(bits)
    assert np.array_equal(va, vb) and np.array_equal(la, lb)
    c = pkg.ScanEngine(plan, u, precision="c64f32", batch_tile=4)
    assert a.launch_count(11) == a.launch_count(8) + c.launch_count(3)
