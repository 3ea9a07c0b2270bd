"""Kernels that start while their predecessor runs (chained_start, scan_device.cuh).

CPU: what an earlier kernel of a chain writes (tables, weights, flags, maxima, Gram partials)
is read with coherent loads.  CUDA defines the read-only path (__ldg, const __restrict__)
only for data that nobody writes while the kernel lives, and an early start puts the
predecessor's writes into just that time.

GPU: sweeps whose kernels start early (tables of a small tile, up to 64 MiB) against the same
sweeps without (a tile whose tables are larger), bitwise, repeated.
"""
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "rgs70-classical-challenge_b200" / "csrc"
# Plan data and the caller's inputs: complete before the first kernel of a chain starts.
CONSTANT = {"T", "tables", "U", "uniforms"}


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _kernels():
    """(name, parameters, body) of every kernel that calls chained_start."""
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        code = _code(path)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*"
                             r"\(([^)]*)\)\s*\{", code):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(code[end], 0)
                end += 1
            body = code[m.end():end]
            if "chained_start();" in body:
                yield m.group(1), [p.strip() for p in m.group(2).split(",")], body


def test_chained_kernels_read_coherently():
    names = set()
    for name, params, body in _kernels():
        names.add(name)
        for p in params:
            if "*" in p and "const" in p and "__restrict__" in p:
                assert p.split()[-1].lstrip("*") in CONSTANT, (name, p)
        assert "__ldg" not in body, name
    assert names == {"scan_row_kernel", "scan_pair_kernel", "chain_gram_kernel", "chain_decide_kernel"}
    device = _code(CSRC / "scan_device.cuh")
    loads = re.findall(r"#define RGS_LD\(p\) (.*)", device)
    assert loads and not any("__ldg" in x for x in loads)
    for m in re.finditer(r"__ldg\(([^;]*);", device + _code(CSRC / "scan_row.cuh") + _code(CSRC / "scan_pair.cuh")):
        assert re.match(r"(T\b|reinterpret_cast<const ulonglong2\*>\(T2\))", m.group(1)), m.group(0)


def _plan(pkg, rank, seed):
    while True:
        seed += 1
        rng = np.random.default_rng(seed)
        n = 36
        g = pkg.instances.degree_at_most3(n, rng)
        order = rng.permutation(n).tolist()
        e = pkg.edges_from_graph(g)
        if max(pkg.rank_profile(n, e, order)) == rank:
            plan = pkg.ScanPlan(n, e, order)
            if plan.pairs:
                return n, g, pkg.instances.haar_su2(n, rng), order, plan


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["c64", "c64f32", "c128"])
@pytest.mark.parametrize("rank", [13, 17])
def test_early_start_changes_nothing(pkg, rank, precision):
    """Rank 17: the largest tile's peak tables exceed 64 MiB, those of tiles 1 to 16 do not."""
    n, g, u, order, plan = _plan(pkg, rank, 10 * rank)
    rng = np.random.default_rng(rank)
    bits = pkg.instances.uniform_bits(150, n, rng)
    whole = pkg.ScanEngine(plan, u, precision=precision, batch_tile=pkg.max_batch_tile(precision))
    assert whole.launch_count(150) > n // 2
    ref = whole.sweep_bits(bits)
    for tile in (1, 4, 16):
        eng = pkg.ScanEngine(plan, u, precision=precision, batch_tile=tile)
        for _ in range(4):
            v, l = eng.sweep_bits(bits)
            assert np.array_equal(v, ref[0]) and np.array_equal(l, ref[1]), tile
    uni = rng.random((90, n))
    cap = 64 if precision == "c128" else 128
    bits, p, logp = pkg.ChainSampler(g, u, order, precision=precision, plan=plan, batch_tile=cap).sample(90, uniforms=uni)
    for tile in (4, 16):
        cs = pkg.ChainSampler(g, u, order, precision=precision, plan=plan, batch_tile=tile)
        for _ in range(4):
            b, q, lq = cs.sample(90, uniforms=uni)
            assert np.array_equal(b, bits) and np.array_equal(q, p) and np.abs(lq - logp).max() < 1e-9, tile
