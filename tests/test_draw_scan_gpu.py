"""The draw's inverse CDF (one block: chunk sums, shuffle scan, search) where chunks are
uneven or empty: few tiles and many, uniforms at 0, just below 1, and on both sides of
cumulative masses.

The drawn index is the first whose cumulative probability in float64 exceeds the uniform;
uniforms are kept 1e-9 away from every boundary that could move by rounding (sums of at
most 2^15 masses or 2^12 values, each relative 2^-52).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Fixed:
    def __init__(self, us):
        self.us = list(us)

    def random(self):
        return self.us.pop(0)


@pytest.mark.parametrize("m", [6, 12, 13, 16, 24])
def test_draw_matches_cumulative_sum(pkg, m):
    from oracle import graph_state as gs
    rng = np.random.default_rng(m)
    while True:
        g = pkg.instances.dense(2 * m, rng)
        A, B = list(range(m)), list(range(m, 2 * m))
        if gs.gf2rank(g[np.ix_(B, A)]) == m:
            break
    u = pkg.instances.haar_su2(2 * m, rng)
    u[B] = u[B[0]]
    s = pkg.ConditionalSampler(g, u, A, B, deferred=False)
    s.compute(rng.integers(0, 2, m).tolist())
    v = s.state.cpu().numpy()
    p = v.real.astype(np.float64) ** 2 + v.imag.astype(np.float64) ** 2
    tiles, norm, tb, nt = s.masses()
    ct = np.cumsum(tiles)
    hits = 0
    for u1 in [0.0, 1 - 2.0 ** -53, *rng.random(12), *(ct[rng.integers(0, nt, 6)] / ct[-1] + 1e-8),
               *(ct[rng.integers(0, nt, 6)] / ct[-1] - 1e-8)]:
        u1 = float(min(max(u1, 0.0), 1 - 2.0 ** -53))
        u2 = float(rng.random())
        tile = min(int(np.searchsorted(ct, u1 * ct[-1], side="right")), nt - 1)
        q = np.cumsum(p[tile << tb:(tile + 1) << tb])
        within = min(int(np.searchsorted(q, u2 * q[-1], side="right")), len(q) - 1)
        near = min(np.abs(ct - u1 * ct[-1]).min(), np.abs(q - u2 * q[-1]).min() / q[-1]) < 1e-9
        idx, pa, nrm = s.draw(_Fixed([u1, u2, 0.5]))
        assert abs(nrm - ct[-1]) < 1e-12
        if u1 < 1 - 2.0 ** -53 and not near:
            assert idx == (tile << tb) + within, (u1, u2)
            hits += 1
        assert p[idx] > 0 and abs(pa - p[idx]) <= 1e-15
    assert hits >= 8
