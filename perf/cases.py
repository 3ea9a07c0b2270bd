"""The calls whose speed matters to a program that uses this package, as timed cases.

Kinds of call, each through a public entry point:

* ``amplitudes``  p(x) of given bitstrings by the scan: ``ScanOracle.amplitudes`` on host
  bitstrings for a single string, ``ScanEngine.run_bits`` on device bitstrings for batches;
* ``samples``     exact Born samples by the chain rule (``ChainSampler.sample_device``);
* ``marginals``   conditionals of given bitstrings (``ChainSampler.marginals``);
* ``batch``       many uneven small instances in one launch (``ResidentBatch``);
* ``conditional`` the Fourier-cut conditional state and one draw (``ConditionalSampler``);
* ``made``        loss and gradients of the proposal network (``MadeProposal.gradients``).

Graphs and scan orders belong to a case; gates, bitstrings, sampler seeds and network
weights come from the seed.  Results that carry the rounding of complex64 tables are kept
as a program stores them: complex64 amplitudes, float32 log-probabilities.
"""
import math

import numpy as np
import torch

import __graft_entry__

rgs = __graft_entry__.package()

LN2 = math.log(2.0)
SEARCH_ITERATIONS = 20000


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # One string in complex128: the latency of ScanOracle.amplitude(s), and of every
        # FP64 recheck of a single decision.
        dict(name="one_string_n24", kind="amplitudes", graph="reg3", n=24, graph_seed=24, order="random",
             order_seed=1004, precision="c128", count=1),
        # The CPU-checkable workload: 4096 uniform strings at n = 24, default precision.
        dict(name="strings_n24", kind="amplitudes", graph="reg3", n=24, graph_seed=24, order="random",
             order_seed=1003, precision="c64", count=4096),
        # The throughput workload of the benchmark, bulk precision: rank 20.
        dict(name="strings_n40_bulk", kind="amplitudes", graph="reg3", n=40, graph_seed=40, order="random",
             order_seed=1582, precision="c64f32", count=16384),
        # Its complex128 recheck, over a count that no batch tile divides.
        dict(name="strings_n40_recheck", kind="amplitudes", graph="reg3", n=40, graph_seed=40, order="random",
             order_seed=1582, precision="c128", count=5000),
        # Full-size circuits with the order search first, as the package advises: rank 11.
        dict(name="strings_n70_searched", kind="amplitudes", graph="deg3", n=70, graph_seed=70, order="searched",
             order_seed=1001, precision="c64f32", count=16384),
        # Large tables and few strings (rank 26, 0.5 GiB per table and string).
        dict(name="strings_n70_rank26", kind="amplitudes", graph="deg3", n=70, graph_seed=70, order="random",
             order_seed=2, precision="c64f32", count=11),
        # 1000 exact samples of the n = 24 workload, default precision.
        dict(name="samples_n24", kind="samples", graph="reg3", n=24, graph_seed=24, order="random",
             order_seed=1003, precision="c64", count=1000),
        # Exact samples at rank 20, bulk precision.
        dict(name="samples_n40", kind="samples", graph="reg3", n=40, graph_seed=40, order="random",
             order_seed=1582, precision="c64f32", count=512),
        # Conditionals of given strings: the training targets of the proposal network.
        dict(name="marginals_n56", kind="marginals", graph="deg3", n=56, graph_seed=56, order="searched",
             order_seed=5, precision="c64f32", count=8192),
        # Uneven instances, amplitudes and samples of each, in one launch.
        dict(name="batch_256", kind="batch", instances=256, n_min=20, n_max=36, strings=256, samples=64,
             graph_seed=2026, precision="c64"),
        # The conditional sampler's state and draw (2^27 complex64 values).
        dict(name="conditional_m27", kind="conditional", m=27, graph_seed=1027),
        # One training batch of the proposal network (2 x 512 hidden units).
        dict(name="made_n56", kind="made", n=56, hidden=512, rows=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scan_case(rng, kind, sizes, most):
    """A graph, an order and a count of the listed ranges; ``most`` bounds table entries x
    strings, so that a drawn case stays below the largest listed ones."""
    while True:
        graph = rng.choice(["reg3", "deg3", "er3"])
        searched = rng.random() < 0.5
        n = rng.randint(20, 70 if searched else 56)
        n += n % 2 if graph == "reg3" else 0
        case = dict(kind=kind, graph=graph, n=n, graph_seed=rng.randint(1, 10 ** 6),
                    order="searched" if searched else "random", order_seed=rng.randint(1, 10 ** 6),
                    precision=rng.choice(["c64", "c64f32", "c128"]), count=_log_int(rng, *sizes))
        g, order = _instance(case)
        ranks = rgs.rank_profile(n, rgs.edges_from_graph(g), order)
        cost = sum(1 << r for r in ranks) * (2 if case["precision"] == "c128" else 1)
        case["count"] = min(case["count"], int(most // cost))
        if case["count"] >= 1 and max(ranks) <= 26:
            return case


def draw(rng):
    kind = rng.choice(["amplitudes", "amplitudes", "amplitudes", "samples", "marginals", "batch", "conditional",
                       "made"])
    if kind == "amplitudes":
        return _scan_case(rng, kind, (1, 16384), 2.0e10)
    if kind == "samples":
        return _scan_case(rng, kind, (1, 2048), 1.0e9)
    if kind == "marginals":
        return _scan_case(rng, kind, (64, 8192), 1.0e9)
    if kind == "batch":
        lo = rng.randint(16, 30)
        return dict(kind=kind, instances=_log_int(rng, 8, 256), n_min=lo, n_max=lo + rng.randint(0, 12),
                    strings=_log_int(rng, 1, 256), samples=rng.randint(0, 64), graph_seed=rng.randint(1, 10 ** 6),
                    precision=rng.choice(["c64", "c64", "c64f32", "c128"]))
    if kind == "conditional":
        return dict(kind=kind, m=rng.randint(13, 27), graph_seed=rng.randint(1, 10 ** 6))
    return dict(kind="made", n=rng.randint(16, 70), hidden=rng.choice([128, 256, 384, 500, 512, 768]),
                rows=_log_int(rng, 100, 8192))


# ------------------------------------------------------------------- inputs of a case
def _graph(name, n, rng):
    return {"reg3": rgs.instances.regular3, "er3": rgs.instances.erdos_renyi,
            "deg3": rgs.instances.degree_at_most3}[name](n, rng)


def _instance(case):
    """Graph and scan order of a scan case (the same for every seed)."""
    n = case["n"]
    g = _graph(case["graph"], n, np.random.default_rng(case["graph_seed"]))
    order = np.random.default_rng(case["order_seed"]).permutation(n).tolist()
    if case["order"] == "searched":
        order, _, _ = rgs.search_order(n, rgs.edges_from_graph(g), order, iterations=SEARCH_ITERATIONS, seed=1,
                                       threads=1)
    return g, order


def _batch_instances(case):
    rng = np.random.default_rng(case["graph_seed"])
    out = []
    for _ in range(case["instances"]):
        n = int(rng.integers(case["n_min"], case["n_max"] + 1))
        g = _graph("er3", n, rng)
        order, _, _ = rgs.search_order(n, rgs.edges_from_graph(g), rng.permutation(n).tolist(), iterations=2000,
                                       seed=1, threads=1)
        out.append((g, order))
    return out


def _cut(case):
    """A dense graph on 2m vertices whose cut A = 0..m-1, B = m..2m-1 has full rank."""
    m, rng = case["m"], np.random.default_rng(case["graph_seed"])
    A, B = list(range(m)), list(range(m, 2 * m))
    while True:
        g = rgs.instances.dense(2 * m, rng)
        if _gf2_rank(g[np.ix_(B, A)]) == m:
            return g, A, B


def _gf2_rank(a):
    rows = [int("".join(map(str, r)), 2) for r in np.asarray(a)]
    rank = 0
    while rows:
        p = rows.pop()
        if p:
            rank += 1
            low = p & -p
            rows = [r ^ p if r & low else r for r in rows]
    return rank


def _scan_inputs(case, seed):
    rng = np.random.default_rng([seed, case["n"], case["count"]])
    u = rgs.instances.haar_su2(case["n"], rng)
    bits = rgs.instances.uniform_bits(case["count"], case["n"], rng)
    return u, bits, int(rng.integers(1, 2 ** 62))


def _batch_inputs(case, seed, insts):
    rng = np.random.default_rng([seed, 7])
    return [(rgs.instances.haar_su2(len(g), rng), rgs.instances.uniform_bits(case["strings"], len(g), rng),
             int(rng.integers(1, 2 ** 62))) for g, _ in insts]


def _conditional_inputs(case, seed):
    rng = np.random.default_rng([seed, case["m"]])
    u = rgs.instances.haar_su2(2 * case["m"], rng)
    u[case["m"]:] = u[case["m"]]     # identical gates on B, the sampler's production form
    return u, rng.integers(0, 2, case["m"]).tolist(), rng


def _made_inputs(case, seed):
    n, h = case["n"], case["hidden"]
    rng = np.random.default_rng([seed, n, h])
    masks = rgs.proposal.made_masks(n, h)
    w = [(rng.normal(size=m.shape) * math.sqrt(2.0 / max(1.0, m.sum(axis=1).mean())) * m).astype(np.float32)
         for m in masks]
    b = [(0.1 * rng.normal(size=m.shape[0])).astype(np.float32) for m in masks]
    x = rng.integers(0, 2, (case["rows"], n)).astype(np.float32)
    target = rng.beta(0.8, 0.8, (case["rows"], n)).astype(np.float32)
    return masks, w, b, x, target


# -------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", 0)
    if kind in ("amplitudes", "samples", "marginals"):
        g, order = _instance(case)
        u, bits, sampler_seed = _scan_inputs(case, seed)
        s = dict(kind=kind, n=case["n"], count=case["count"])
        if kind == "amplitudes":
            s["oracle"] = rgs.ScanOracle(g, u, order, precision=case["precision"])
            s["bits"] = bits
            if case["count"] > 1:
                s["d_bits"] = torch.from_numpy(rgs.pack_bits(bits, case["n"]).view(np.int64)).to(dev)
                s["value"], s["logscale"] = s["oracle"].engine.out_tensors(case["count"])
        else:
            s["sampler"] = rgs.ChainSampler(g, u, order, precision=case["precision"])
            s["bits"], s["seed"] = bits, sampler_seed
        return s
    if kind == "batch":
        insts = _batch_instances(case)
        rb = rgs.ResidentBatch(case["precision"])
        K, S, nI = case["strings"], case["samples"], len(insts)
        vdt = torch.complex128 if case["precision"] == "c128" else torch.complex64
        s = dict(kind=kind, batch=rb, value=torch.zeros(nI * K, dtype=vdt, device=dev),
                 logscale=torch.zeros(nI * K, dtype=torch.float64, device=dev),
                 sbits=torch.zeros((nI * S, 2), dtype=torch.int64, device=dev),
                 svalue=torch.zeros(nI * S, dtype=vdt, device=dev),
                 slogscale=torch.zeros(nI * S, dtype=torch.float64, device=dev),
                 slogp=torch.zeros(nI * S, dtype=torch.float64, device=dev))
        ns, keep = [], []
        for k, ((g, order), (u, bits, sd)) in enumerate(zip(insts, _batch_inputs(case, seed, insts))):
            n = len(g)
            plan = rgs.ScanPlan(n, rgs.edges_from_graph(g), order)
            du = torch.from_numpy(u.view(np.float64).reshape(-1).copy()).to(dev)
            db = torch.from_numpy(rgs.pack_bits(bits, n).view(np.int64)).to(dev)
            a, b, c, d = k * K, (k + 1) * K, k * S, (k + 1) * S
            rb.add_device(plan, du, db, s["value"][a:b], s["logscale"][a:b], S, sd, s["sbits"][c:d],
                          s["svalue"][c:d], s["slogscale"][c:d], s["slogp"][c:d])
            ns += [n]
            keep += [(plan, du, db)]
        s["keep"] = keep
        s["shift"] = torch.tensor(ns, dtype=torch.float64, device=dev) * (0.5 * LN2)
        rb.tune()
        return s
    if kind == "conditional":
        g, A, B = _cut(case)
        u, outb, rng = _conditional_inputs(case, seed)
        return dict(kind=kind, sampler=rgs.ConditionalSampler(g, u, A, B), outb=outb, rng=rng)
    masks, w, b, x, target = _made_inputs(case, seed)
    net = rgs.MadeProposal(case["n"], hidden=case["hidden"], seed=0)
    for i in range(3):
        net.w[i].copy_(torch.from_numpy(w[i]))
        net.b[i].copy_(torch.from_numpy(b[i]))
        net.wb[i].copy_((net.w[i] * net.masks[i]).to(torch.bfloat16))
    return dict(kind=kind, net=net, x=torch.from_numpy(x).to(dev).to(torch.bfloat16),
                target=torch.from_numpy(target).to(dev))


def _amplitude(value, logscale, shift):
    """value * exp(logscale) * 2^(-n/2) in the precision of the tables; shift = n ln(2) / 2."""
    return value * torch.exp(logscale - shift).to(value.real.dtype)


def _stored(x, precision_of):
    """Log-probabilities from complex64 tables are stored as float32."""
    return x if precision_of.dtype == torch.complex128 else x.to(torch.float32)


def run(state):
    kind = state["kind"]
    if kind == "amplitudes":
        if "d_bits" not in state:
            return state["oracle"].amplitudes(state["bits"])
        state["oracle"].engine.run_bits(state["d_bits"], state["value"], state["logscale"])
        return _amplitude(state["value"], state["logscale"], 0.5 * LN2 * state["n"])
    if kind == "samples":
        bits, value, logscale, logp = state["sampler"].sample_device(state["count"], seed=state["seed"])
        return bits, _amplitude(value, logscale, 0.5 * LN2 * state["n"]), _stored(logp, value)
    if kind == "marginals":
        cond, logp, p = state["sampler"].marginals(state["bits"])
        if state["sampler"].precision != "c128":
            logp, p = logp.astype(np.float32), p.astype(np.float32)
        return cond, logp, p
    if kind == "batch":
        state["batch"].run(check=False)
        out, shift = [], state["shift"]
        for v, ls in ((state["value"], state["logscale"]), (state["svalue"], state["slogscale"])):
            if v.numel():
                out.append(_amplitude(v.view(len(shift), -1), ls.view(len(shift), -1), shift[:, None]))
        return out + [state["sbits"], _stored(state["slogp"], state["svalue"])]
    if kind == "conditional":
        s = state["sampler"]
        s.compute(state["outb"])
        index, pa, norm = s.draw(state["rng"])
        return s.state, index, pa, norm
    loss, grads = state["net"].gradients(state["x"], state["target"])
    return [loss] + grads


# --------------------------------------------------------------------- work of a pass
def _scan_flops(ranks):
    """One complex multiply-add (8 flops) per weight and table entry of every position."""
    r_in = [0] + list(ranks[:-1])
    return 8.0 * sum(2 * (1 << max(a, b)) for a, b in zip(r_in, ranks))


def work(case):
    kind = case["kind"]
    if kind in ("amplitudes", "samples", "marginals"):
        n, c = case["n"], case["count"]
        g, order = _instance(case)
        ranks = rgs.rank_profile(n, rgs.edges_from_graph(g), order)
        es = 16 if case["precision"] == "c128" else 8
        out = {"amplitudes": es, "samples": 16 + 2 * es, "marginals": 4 * n + es}[kind]
        read = 0 if kind == "samples" else 16
        # A sample also needs both branch masses of every position.
        return {"bytes": float(64 * n + c * (read + out)),
                "flops": c * _scan_flops(ranks) * (1 if kind == "amplitudes" else 2)}
    if kind == "batch":
        flops = nbytes = 0.0
        es = 16 if case["precision"] == "c128" else 8
        for g, order in _batch_instances(case):
            f = _scan_flops(rgs.rank_profile(len(g), rgs.edges_from_graph(g), order))
            flops += f * (case["strings"] + 2 * case["samples"])
            nbytes += 64 * len(g) + case["strings"] * (16 + es) + case["samples"] * (16 + 2 * es)
        return {"bytes": nbytes, "flops": flops}
    if kind == "conditional":
        m = case["m"]
        # The state is written once; Walsh butterflies (4 flops a value and bit) and 2x2
        # products (14 flops a value and bit).
        return {"bytes": 8.0 * 2 ** m, "flops": float(m * 18 * 2 ** m)}
    n, h, r = case["n"], case["hidden"], case["rows"]
    params = n * h + h * h + h * n
    return {"bytes": float(2 * r * n + 4 * r * n + 2 * params + 4 * (params + 2 * h + n)),
            "flops": float(2 * r * (2 * n * h + h * h) + 2 * r * (n * h + 2 * (n * h + h * h)))}


# ----------------------------------------------------------- the same, in 64 bits
def _dev():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _greedy_order(g):
    """A vertex order with a small boundary: next, the vertex that leaves the fewest
    unprocessed vertices adjacent to processed ones."""
    n = len(g)
    nb = [set(np.flatnonzero(g[v]).tolist()) for v in range(n)]
    best = None
    for start in range(n):
        todo, edge, order, peak = set(range(n)), set(), [], 0
        v = start
        while True:
            todo.discard(v)
            edge = (edge | (nb[v] & todo)) - {v}
            order.append(v)
            peak = max(peak, len(edge))
            if not todo:
                break
            v = min(edge or todo, key=lambda w: (len(nb[w] & todo - edge), w))
        if best is None or peak < best[0]:
            best = (peak, order)
    return best[1]


def _peak(g, order):
    todo, edge, peak = set(range(len(g))), set(), 0
    for v in order:
        todo.discard(v)
        edge = (edge | (set(np.flatnonzero(g[v]).tolist()) & todo)) - {v}
        peak = max(peak, len(edge))
    return peak


def _sweep64(g, u, order, bits=None, uniforms=None):
    """Amplitudes of strings by a vertex-by-vertex sum in complex128: E holds one axis per
    unprocessed vertex adjacent to a processed one, the parity of its processed neighbours.
    ``bits`` [B, n] given, or drawn position by position with ``uniforms`` [B, n] from the
    branch masses.  Returns (amplitude, log p, p(x_v = 1 | prefix) by position)."""
    dev, n = _dev(), len(g)
    ud = torch.from_numpy(np.asarray(u, np.complex128)).to(dev)
    src = bits if uniforms is None else uniforms
    chunk = max(1, (1 << 25) >> _peak(g, order))
    amps, lps, conds = [], [], []
    for c0 in range(0, len(src), chunk):
        part = torch.as_tensor(np.ascontiguousarray(src[c0:c0 + chunk])).to(dev)
        B = len(part)
        E = torch.ones((B, 1), dtype=torch.complex128, device=dev)
        axes, todo = [], set(range(n))
        lp = torch.zeros(B, dtype=torch.float64, device=dev)
        cond = torch.zeros((B, n), dtype=torch.float64, device=dev)
        for j, v in enumerate(order):
            todo.discard(v)
            if v in axes:
                i = axes.index(v)
                t = E.view(B, 2 ** i, 2, -1)
                a0, a1 = (t[:, :, 0] + t[:, :, 1]).reshape(B, -1), (t[:, :, 0] - t[:, :, 1]).reshape(B, -1)
                axes.pop(i)
            else:
                a0 = a1 = E
            near = [w for w in np.flatnonzero(g[v]).tolist() if w in todo]
            flip = sum(1 << (len(axes) - 1 - axes.index(w)) for w in near if w in axes)
            new = [w for w in near if w not in axes]
            if flip:
                a1 = a1[:, torch.arange(a1.shape[1], device=dev) ^ flip]
            g00 = (a0.real ** 2 + a0.imag ** 2).sum(1)
            g11 = (a1.real ** 2 + a1.imag ** 2).sum(1)
            g01 = torch.zeros_like(g00, dtype=torch.complex128) if new else (a0 * a1.conj()).sum(1)
            mass = [g00 * abs(u[v, x, 0]) ** 2 + g11 * abs(u[v, x, 1]) ** 2 +
                    2 * (g01 * complex(u[v, x, 0] * np.conj(u[v, x, 1]))).real for x in (0, 1)]
            cond[:, j] = mass[1] / (mass[0] + mass[1])
            x = part[:, v].long() if uniforms is None else \
                (part[:, j] * (mass[0] + mass[1]) >= mass[0]).long()
            lp += torch.log(torch.where(x == 1, cond[:, j], 1 - cond[:, j]))
            f = ud[v][x]
            if new:
                E = torch.zeros((B, a0.shape[1], 2 ** len(new)), dtype=torch.complex128, device=dev)
                E[:, :, 0] = f[:, :1] * a0
                E[:, :, -1] = f[:, 1:] * a1
                E = E.view(B, -1)
                axes += new
            else:
                E = f[:, :1] * a0 + f[:, 1:] * a1
        amps.append(E[:, 0] * 2.0 ** (-0.5 * n))
        lps.append(lp)
        conds.append(cond)
    return torch.cat(amps), torch.cat(lps), torch.cat(conds)


def _philox_uniforms(seed, count, n):
    """The sampler's uniforms: Philox4x32-10 (Salmon et al. 2011) of (item, position)."""
    m32 = np.uint64(0xFFFFFFFF)
    item = np.repeat(np.arange(count, dtype=np.uint64)[:, None], n, axis=1)
    c = [item & m32, item >> np.uint64(32), np.repeat(np.arange(n, dtype=np.uint64)[None, :], count, axis=0),
         np.zeros((count, n), np.uint64)]
    k = [seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF]
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k[0]), p1 & m32,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k[1]), p0 & m32]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return (((c[0] << np.uint64(32)) | c[1]) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _conditional64(g, u, A, B, outb):
    """psi(x_A | x_B) of the cut in complex128: Walsh transform of the B side's phases and
    gates, read at G_BA a, the A side's phases, then the A gates but the last qubit's."""
    dev, m = _dev(), len(A)
    ud = np.asarray(u, np.complex128)

    def quad(idx, Q):          # sign of sum_{i<j} Q_ij b_i b_j
        acc = torch.zeros(len(idx), dtype=torch.int64, device=dev)
        for i in range(m):
            row = int(sum(int(Q[i, j]) << j for j in range(i)))
            if row:
                w = idx & row
                for s in (16, 8, 4, 2, 1):
                    w = w ^ (w >> s)
                acc ^= ((idx >> i) & 1) & (w & 1)
        return acc

    idx = torch.arange(2 ** m, device=dev)
    v = torch.ones(1, dtype=torch.complex128, device=dev)
    for i in reversed(range(m)):                       # qubit B[i] = bit i
        v = (v[:, None] * torch.from_numpy(ud[B[i], outb[i]]).to(dev)[None, :]).reshape(-1)
    v = v * (1 - 2 * quad(idx, g[np.ix_(B, B)]))
    for i in range(m):
        t = v.view(-1, 2, 2 ** i)
        v = torch.stack((t[:, 0] + t[:, 1], t[:, 0] - t[:, 1]), 1).reshape(-1)
    at = torch.zeros_like(idx)
    for i in range(m):                                 # a_i = 1 adds its B neighbours
        at ^= ((idx >> i) & 1) * int(sum(int(g[B[j], A[i]]) << j for j in range(m)))
    v = v[at] * (1 - 2 * quad(idx, g[np.ix_(A, A)]))
    del at, idx
    for i in range(m - 1):
        U, t = ud[A[i]], v.view(-1, 2, 2 ** i)
        v = torch.stack((complex(U[0, 0]) * t[:, 0] + complex(U[0, 1]) * t[:, 1],
                         complex(U[1, 0]) * t[:, 0] + complex(U[1, 1]) * t[:, 1]), 1).reshape(-1)
    return v * 2.0 ** (-0.5 * m)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("amplitudes", "samples", "marginals"):
        g, order = _instance(case)
        u, bits, sampler_seed = _scan_inputs(case, seed)
        if kind == "amplitudes":
            amp = _sweep64(g, u, _greedy_order(g), bits)[0]
            return amp.cpu().numpy() if case["count"] == 1 else amp
        if 2.0 ** _peak(g, order) * case["count"] * len(g) > 4.0e11:
            return None                                # too long in 64 bits
        if kind == "samples":
            amp, logp, _ = _sweep64(g, u, order, uniforms=_philox_uniforms(sampler_seed, case["count"], len(g)))
            return None, amp, logp
        amp, logp, cond = _sweep64(g, u, order, bits)
        return cond.cpu().numpy(), logp.cpu().numpy(), (amp.abs() ** 2).cpu().numpy()
    if kind == "batch":
        insts = _batch_instances(case)
        amps, samps, logps = [], [], []
        for (g, order), (u, bits, sd) in zip(insts, _batch_inputs(case, seed, insts)):
            amps.append(_sweep64(g, u, order, bits)[0])
            if case["samples"]:
                a, lp, _ = _sweep64(g, u, order, uniforms=_philox_uniforms(sd, case["samples"], len(g)))
                samps.append(a)
                logps.append(lp)
        out = [torch.stack(amps)] + ([torch.stack(samps)] if samps else [])
        return out + [None, torch.cat(logps) if logps else None]
    if kind == "conditional":
        g, A, B = _cut(case)
        u, outb, _ = _conditional_inputs(case, seed)
        return _conditional64(g, u, A, B, outb), None, None, 1.0
    masks, w, b, x, target = _made_inputs(case, seed)
    w, b, m, x, t = ([torch.from_numpy(np.asarray(q, np.float64)).to(_dev()) for q in p]
                     for p in (w, b, masks, [x], [target]))
    x, t, rows = x[0], t[0], case["rows"]
    h1 = torch.relu(x @ w[0].T + b[0])
    h2 = torch.relu(h1 @ w[1].T + b[1])
    z = h2 @ w[2].T + b[2]
    loss = (torch.nn.functional.softplus(z) - t * z).sum() / rows
    dz = (torch.sigmoid(z) - t) / rows
    d2 = (dz @ w[2]) * (h2 > 0)
    d1 = (d2 @ w[1]) * (h1 > 0)
    return [float(loss), d1.T @ x * m[0], d1.sum(0), d2.T @ h1 * m[1], d2.sum(0), dz.T @ h2 * m[2], dz.sum(0)]
