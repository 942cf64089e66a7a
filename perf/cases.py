"""Workloads for timing the framework: each case is one call, or the short
sequence of calls a program makes together, through the public Python entry
points (a2c_gb300.Gpp and a2c_gb300.Batch).

A case names its operation ("op") and its sizes:

  eval       Gpp.eval_device: objective and gradient on device pointers, the
             minimizer callback of a program that keeps its state on the GPU
  eval_host  Gpp.eval: the same from and to host arrays, the call a TAO-style
             host solver makes at every iterate
  lists      Gpp.build_neighbors at new positions, then one evaluation
  skin       Gpp.update_neighbors (the re-filter of skin lists after a small
             move), then one evaluation
  occupancy  the occupancy part of an outer step: chemical potential,
             Dirichlet condition, diffusion, macro results
  minimize   Gpp.minimize for a fixed number of L-BFGS iterations
  batch      Batch.minimize of many uneven lattices, a fixed number of
             iterations

Lattices are fcc Pd with octahedral H sites (cells z, y, x, then the basis;
all Pd, then all H), displaced by N(0, 0.02 A), as the repository's
benchmark and tests make them; here they are drawn by numpy from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import a2c_gb300 as A

A0 = 3.89            # lattice constant [A]
RC = 5.35            # cutoff [A]
KB = 8.6173324e-5    # [eV/K]
W = 1.0 / 12.0       # quadrature weight
PD = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
OCT = np.array([[.5, 0, 0], [0, .5, 0], [0, 0, .5], [.5, .5, .5]])
X_BD, GAMMA_BD = 0.80, -20.75           # Dirichlet occupancy and its chemical potential at 400 K
DT, NU, QM, X_LB, X_UB = 1e-12, 1e13, 0.23, 1e-3, 1.0 - 1e-16


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A unit-cell study or one member of a parameter scan, in the default
        # precision (FP64): the smallest call, all latency.
        dict(name="eval_fp64_512", op="eval", precision="fp64", nx=4, ny=4, nz=4, px=1, py=1, pz=1, T=300.0,
             x=0.05, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # An ordinary thin film in FP64: odd edges, free surfaces in z, uneven widths.
        dict(name="eval_fp64_film_10k", op="eval", precision="fp64", nx=13, ny=11, nz=9, px=1, py=1, pz=0, T=350.0,
             x=0.30, sigma_lo=0.08, sigma_hi=0.14, nucleus=0),
        # The evaluator-throughput lattice of the benchmark in FP64 (the parity form at full size).
        dict(name="eval_fp64_262k", op="eval", precision="fp64", nx=32, ny=32, nz=32, px=1, py=1, pz=1, T=300.0,
             x=0.05, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # The smallest mixed-precision call.
        dict(name="eval_mixed_512", op="eval", precision="mixed", nx=4, ny=4, nz=4, px=1, py=1, pz=1, T=300.0,
             x=0.05, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # A host solver's callback on an ordinary film: pageable host arrays in and out.
        dict(name="eval_host_mixed_film_34k", op="eval_host", precision="mixed", nx=19, ny=17, nz=13, px=1, py=1,
             pz=0, T=300.0, x=0.10, sigma_lo=0.08, sigma_hi=0.14, nucleus=0),
        # The benchmark's headline workload, at the tile its tuner settles on.
        dict(name="eval_mixed_262k", op="eval", precision="mixed", nx=32, ny=32, nz=32, px=1, py=1, pz=1, T=300.0,
             x=0.05, sigma_lo=0.1, sigma_hi=0.1, nucleus=0, tps=2, rho_block=512, grad_block=256),
        # The largest configuration: the hydride nucleus at 64^3 cells (2,097,152 sites), library defaults.
        dict(name="eval_mixed_2m", op="eval", precision="mixed", nx=64, ny=64, nz=64, px=1, py=1, pz=1, T=300.0,
             x=0.02, sigma_lo=0.1, sigma_hi=0.1, nucleus=1),
        # A list rebuild at new positions before the next solve.
        dict(name="lists_262k", op="lists", precision="mixed", nx=32, ny=32, nz=32, px=1, py=1, pz=1, T=300.0,
             x=0.05, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # The per-step list update of a DMD loop with a skin, on a slab.
        dict(name="skin_slab_92k", op="skin", precision="mixed", nx=24, ny=24, nz=20, px=1, py=1, pz=0, T=400.0,
             x=0.01, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # The occupancy update that ends an outer step of the coupled-DMD slab.
        dict(name="occupancy_slab_111k", op="occupancy", precision="mixed", nx=24, ny=24, nz=24, px=1, py=1, pz=0,
             T=400.0, x=0.10, sigma_lo=0.1, sigma_hi=0.1, nucleus=0),
        # Whole call: the first 20 iterations of the nucleus minimization at 32^3 cells.
        dict(name="minimize_nucleus_262k", op="minimize", precision="mixed", nx=32, ny=32, nz=32, px=1, py=1, pz=1,
             T=300.0, x=0.02, sigma_lo=0.1, sigma_hi=0.1, nucleus=1, iters=20),
        # Whole call: uneven independent lattices minimized together.
        dict(name="batch_24", op="batch", precision="mixed", n=24, edge_lo=4, edge_hi=14, iters=12),
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm,
    any edges, any periodicity."""
    op = rng.choice(["eval", "eval", "eval", "eval_host", "lists", "skin", "occupancy", "minimize", "batch"])
    precision = rng.choice(["fp64", "mixed"]) if op in ("eval", "eval_host") else "mixed"
    if op == "batch":
        lo = rng.randint(4, 7)
        return dict(op=op, precision=precision, n=int(round(math.exp(rng.uniform(math.log(3), math.log(24))))),
                    edge_lo=lo, edge_hi=rng.randint(lo + 1, 14), iters=rng.randint(4, 12))
    top = {"eval": 200_000 if precision == "fp64" else 1_000_000, "eval_host": 60_000, "lists": 250_000,
           "skin": 250_000, "occupancy": 200_000, "minimize": 150_000}[op]
    sites = math.exp(rng.uniform(math.log(900), math.log(top)))
    edge = (sites / 8.0) ** (1.0 / 3.0)
    n = [max(4, int(round(edge * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(2)]
    n.append(max(4, int(round(sites / (8 * n[0] * n[1])))))
    per = [1, 1, 0] if op == "occupancy" else [int(rng.random() < 0.7) for _ in range(3)]
    lo = rng.choice([0.08, 0.1])
    c = dict(op=op, precision=precision, nx=n[0], ny=n[1], nz=n[2], px=per[0], py=per[1], pz=per[2],
             T=float(rng.randrange(200, 601, 50)), x=round(rng.uniform(0.02, 0.6), 3), sigma_lo=lo,
             sigma_hi=rng.choice([lo, 0.14]), nucleus=0)
    if op == "minimize":
        c["iters"] = rng.randint(3, 20)
    return c


# ------------------------------------------------------------------- inputs
def _lattice(n, x, sigma, nucleus, rng):
    """(X 4N, xH, box, nPd, nH): positions and widths, H occupancies."""
    nx, ny, nz = n
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    cell = np.stack([i, j, k], -1).reshape(-1, 1, 3).astype(np.float64)
    q = np.concatenate([(A0 * (cell + PD)).reshape(-1, 3), (A0 * (cell + OCT)).reshape(-1, 3)])
    half = len(q) // 2
    box = (A0 * nx, A0 * ny, A0 * nz)
    if nucleus:  # hydride nucleus: x = 0.60 inside a tanh interface 5 A wide, radius 80 A at 64 cells
        r = np.linalg.norm(q[half:] - 0.5 * np.array(box), axis=1)
        xH = x + (0.60 - x) * 0.5 * (1.0 - np.tanh((r - 80.0 * nx / 64.0) / 5.0))
    else:
        xH = np.clip(x + rng.uniform(-0.01, 0.01, half), X_LB, X_UB)
    X = np.empty((len(q), 4))
    X[:, :3] = q + 0.02 * rng.standard_normal(q.shape)
    X[:, 3] = sigma[0] if sigma[0] == sigma[1] else rng.uniform(sigma[0], sigma[1], len(q))
    return X.reshape(-1), xH, box, half, half


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    X, xH, box, nPd, nH = _lattice((case["nx"], case["ny"], case["nz"]), case["x"],
                                   (case["sigma_lo"], case["sigma_hi"]), case["nucleus"], rng)
    periodic = (case["px"], case["py"], case["pz"])
    inp = dict(X=X, xH=xH, box=box, nPd=nPd, nH=nH, periodic=periodic, T=case["T"])
    if case["op"] == "skin":  # the positions the candidates were made at
        inp["X0"] = X
        X = X.copy().reshape(-1, 4)
        X[:, :3] += np.clip(0.04 * rng.standard_normal((len(X), 3)), -0.12, 0.12)
        inp["X"] = X.reshape(-1)
    if case["op"] == "occupancy":  # the lowest H layer is held at the Dirichlet occupancy
        z = (X.reshape(-1, 4)[nPd:, 2])
        inp["bd"] = np.nonzero(z < 0.25 * A0)[0].astype(np.int32)
        inp["xH"] = xH = xH.copy()
        xH[inp["bd"]] = X_BD
        inp["gamma"] = np.full(nH, GAMMA_BD)
        inp["full"] = np.zeros(nH, dtype=np.int32)
    return inp


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["n"] * 1000 + case["edge_lo"])  # the lattices' edges belong to the case
    inst, Xs, xs = [], [], []
    for _ in range(case["n"]):
        e = int(sizes.integers(case["edge_lo"], case["edge_hi"] + 1))
        T = float(rng.uniform(200.0, 600.0))
        X, xH, box, nPd, nH = _lattice((e, e, e), float(rng.uniform(0.02, 0.70)), (0.1, 0.1), 0, rng)
        inst.append(dict(nPd=nPd, nH=nH, T=T, box=box, periodic=(1, 1, 1)))
        Xs.append(X)
        xs.append(xH)
    return inst, np.concatenate(Xs), np.concatenate(xs)


def prepare(case, seed):
    if case["op"] == "batch":
        inst, X, xH = _batch_inputs(case, seed)
        b = A.Batch(inst, precision=case["precision"])
        b.set_occupancy(xH)
        b.build_neighbors(X)
        return dict(case=case, b=b, X=X)
    p = _inputs(case, seed)
    g = A.Gpp(p["nPd"], p["nH"], T=p["T"], box=p["box"], periodic=p["periodic"], precision=case["precision"])
    g.set_occupancy(p["xH"])
    if case["op"] == "skin":
        g.set_neighbor_skin(0.5)
        g.update_neighbors(p["X0"])
    else:
        g.build_neighbors(p["X"])
    if "tps" in case:
        g.set_tile(case["tps"], case["rho_block"], case["grad_block"])
    s = dict(p, case=case, g=g)
    if case["op"] in ("eval", "lists", "skin"):
        s["dX"] = torch.from_numpy(p["X"]).cuda()
        s["dG"] = torch.empty_like(s["dX"])
        s["df"] = torch.empty(1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    if case["op"] == "occupancy":
        g.set_state(p["X"])
    return s


# --------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "batch":
        r = s["b"].minimize(s["X"], max_it=case["iters"], polish=0)
        return {"X": r.X, "fmin": r.fmin, "gnorm": r.gnorm, "iters": r.iters, "nfev": r.nfev}
    g = s["g"]
    if op == "eval":
        g.eval_device(s["dX"].data_ptr(), s["df"].data_ptr(), s["dG"].data_ptr())
        return {"f": s["df"], "G": s["dG"]}
    if op == "eval_host":
        f, G = g.eval(s["X"])
        return {"f": f, "G": G}
    if op in ("lists", "skin"):
        most = g.build_neighbors(s["X"]) if op == "lists" else g.update_neighbors(s["X"])[0]
        g.eval_device(s["dX"].data_ptr(), s["df"].data_ptr(), s["dG"].data_ptr())
        return {"f": s["df"], "G": s["dG"], "most": most, "shells": g.shell_counts()}
    if op == "occupancy":
        gamma, full = g.chem_potential(GAMMA_BD, s["gamma"], s["full"])
        gamma, full = g.apply_dirichlet(s["bd"], GAMMA_BD, X_BD, gamma, full)
        x = g.diffuse(DT, NU, QM, X_LB, X_UB, gamma, full, s["xH"])
        mean, interior = g.macro_results(x, s["bd"])
        return {"gamma": gamma, "full": full, "x": x, "mean": mean, "interior": interior}
    r = g.minimize(s["X"], max_it=case["iters"], polish=0)
    return {"X": r.X, "fmin": r.fmin, "gnorm": r.gnorm, "iters": r.iters, "nfev": r.nfev}


# -------------------------------------------------------------------- work
# Operations one quadrature point of one pair cannot do without (adds,
# multiplies, an FMA as two, roots and exponentials as one), both passes:
# the density needs the radius and one function; the gradient the radius,
# two density derivatives, the pair function with its derivative, and the
# sums.  80 neighbors per bulk site (42 + 38), fewer at free surfaces.
DENSITY_FLOPS, GRADIENT_FLOPS, POINTS, BULK = 15, 45, 12, 80


def _pairs(case):
    n = (case["nx"], case["ny"], case["nz"])
    sites = 8 * n[0] * n[1] * n[2]
    share = 1.0
    for d, p in enumerate((case["px"], case["py"], case["pz"])):
        if not p:
            share *= max(0.3, 1.0 - 0.375 * RC / (A0 * n[d]))
    return sites, sites * BULK * share


def work(case):
    if case["op"] == "batch":
        sizes = np.random.default_rng(case["n"] * 1000 + case["edge_lo"])
        sites = sum(8 * int(sizes.integers(case["edge_lo"], case["edge_hi"] + 1)) ** 3 for _ in range(case["n"]))
        pairs = sites * BULK
    else:
        sites, pairs = _pairs(case)
    evaluation = {"bytes": 80.0 * sites + 4.0 * pairs, "flops": pairs * POINTS * (DENSITY_FLOPS + GRADIENT_FLOPS)}
    if case["op"] in ("lists", "skin"):  # the lists written once, every listed pair tested once
        evaluation["bytes"] += 32.0 * sites + 4.0 * pairs
        evaluation["flops"] += 8.0 * pairs
    if case["op"] == "occupancy":  # densities of all sites, pair sums of the H sites, 12 hops each
        return {"bytes": 60.0 * sites + 6.0 * pairs,
                "flops": pairs * POINTS * DENSITY_FLOPS * 1.5 + 0.5 * sites * 12 * 10}
    if case["op"] in ("minimize", "batch"):  # an evaluation and a step of L-BFGS (5 pairs) per iteration
        step = {"bytes": 32.0 * sites * 20, "flops": 4.0 * sites * 60}
        return {k: case["iters"] * (evaluation[k] + step[k]) for k in evaluation}
    return evaluation


# ------------------------------------------------------------------- exact
# The same quantities in 64 bits with plain torch: analytic derivatives (by
# autograd), pair lists from a cell search written here.
def _f_pd(r):
    y = r / 5.0
    ra = y
    for b, c in ((2.7267629107325706, 1.8716766113599643), (2.50290548851635, 1.668549182690922),
                 (2.0924467509943674, 1.3150372774478005), (1.564328475106985, 0.8987511149780485),
                 (1.009780903403673, 0.5124363774128722), (0.5304054524800665, 0.2169886022464641),
                 (0.1356566408715063, 0.035852347523891395)):
        ra = ra * (y * (y - b) + c)
    v = -0.02972698211669922 + y * (0.6676807403564453 + y * (-255.8965835571289 + y * (
        14673.409149169922 + -2.597301181336601e7 * ra)))
    t = 0.001510569378297 * torch.exp(-0.077976566126292 / 0.001510569378297 * (r - 5.0))
    return torch.where(r > 5.0, t, v)


def _f_h(r):
    t = 0.009986990526578 * torch.exp(-0.013075667086408 / 0.009986990526578 * (r - 5.35))
    return torch.where(r > 5.35, t, 11.0025 * torch.exp(-1.30927 * r))


def _phi_pd(r):
    y = r / 5.0
    v = -79415.24035137112 * (y - 1.0699996145674568) * (y - 1.06015072612581) * (y - 0.42433991011376526) \
        * (y + 0.06169160085238687)
    for b, c in ((2.0586473420376348, 1.0683922574015199), (1.6696359816422877, 0.7337878627470482),
                 (1.1690370066230809, 0.3909805777737639), (0.2635598721249787, 0.033551116514910245)):
        v = v * (y * (y - b) + c)
    v = v + 2 * 0.251546 * _f_pd(r)
    t = -0.016958780164980 * torch.exp(0.089019679316328 / -0.016958780164980 * (r - 5.05))
    return torch.where(r > 5.05, t, v)


def _morse(r, D, a, b, r0, v, d):
    t = v * torch.exp(d / v * (r - 5.35))
    return torch.where(r > 5.35, t, D * (b * torch.exp(-a * (r - r0)) - a * torch.exp(-b * (r - r0))))


def _phi_pdh(r):
    return _morse(r, 0.2494540, 4.82613, 2.13158, 1.50964, -3.353001113951400e-04, 7.147062196813336e-04)


def _phi_h(r):
    return _morse(r, 0.0661496, 3.67263, 1.47797, 2.51980, -0.003702722457147, 0.005465945471933)


def _embed_pd(rho):
    p = rho / 50.0
    y = 295878.9003038662 * (p - 0.20581955357385892) * (p - 0.081228755904399) * p * (p + 0.05298811034615951)
    for b, c in ((2.4242616904962846, 1.4791899886249564), (2.1376274623740064, 1.2169215689822592),
                 (1.6486007989726832, 0.8159825255339774), (1.0749204110338482, 0.42007491336688396),
                 (0.5128056047933808, 0.12468685331167456)):
        y = y * (p * (p - b) + c)
    return y - 50.0 * 0.251546 * p


def _embed_h(rho):
    c, d, a, b, u = 0.000197047, 1.18860, 9.99780, 60.0155, rho + 0.0540638
    return -c * (u ** (2 + d) / (2 + d) - (a + b) / (1 + d) * u ** (1 + d) + a * b / d * u ** d) + 0.0296604 * rho


def _wrap(d, box, periodic):
    for k in range(3):
        if periodic[k]:
            d[..., k] -= box[k] * torch.round(d[..., k] / box[k])
    return d


def _pair_list(q, box, periodic):
    """Unordered pairs (i, j) within the cutoff."""
    n, dev = len(q), q.device
    cells, lo, ext = [], [], []
    for k in range(3):
        a = 0.0 if periodic[k] else float(q[:, k].min())
        e = box[k] if periodic[k] else float(q[:, k].max()) - a
        lo.append(a)
        ext.append(max(e, 1e-9))
        cells.append(max(1, int(e / (RC + 1e-3))))
    if n <= 12000 or any(periodic[k] and cells[k] < 3 for k in range(3)):
        out = []
        step = max(1, 40_000_000 // n)
        for a in range(0, n, step):
            d = _wrap(q[a:a + step, None, :] - q[None, :, :], box, periodic)
            i, j = torch.nonzero((d * d).sum(-1) <= RC * RC, as_tuple=True)
            i = i + a
            keep = i < j
            out.append(torch.stack([i[keep], j[keep]]))
        return torch.cat(out, 1)
    c = []
    for k in range(3):
        t = (q[:, k] - lo[k]) / ext[k]
        t = t - torch.floor(t) if periodic[k] else t
        c.append((t * cells[k]).long().clamp_(0, cells[k] - 1))
    cid = (c[2] * cells[1] + c[1]) * cells[0] + c[0]
    order = torch.argsort(cid)
    count = torch.bincount(cid, minlength=cells[0] * cells[1] * cells[2])
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    slot = torch.full((len(count), cap), -1, dtype=torch.long, device=dev)
    rank = torch.arange(n, device=dev) - start[cid[order]]
    slot[cid[order], rank] = order
    ids = torch.arange(len(count), device=dev)
    cx, cy, cz = ids % cells[0], (ids // cells[0]) % cells[1], ids // (cells[0] * cells[1])
    out = []
    step = max(1, 30_000_000 // (cap * cap))
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) < (0, 0, 0):
                    continue
                o, ok = [], torch.ones_like(cx, dtype=torch.bool)
                for v, s, k in ((cx, dx, 0), (cy, dy, 1), (cz, dz, 2)):
                    w = v + s
                    if not periodic[k]:
                        ok &= (w >= 0) & (w < cells[k])
                    o.append(w % cells[k])
                other = (o[2] * cells[1] + o[1]) * cells[0] + o[0]
                home = ids[ok]
                for a in range(0, len(home), step):
                    p, r = slot[home[a:a + step]], slot[other[home[a:a + step]]]
                    d = _wrap(q[p.clamp_min(0)][:, :, None, :] - q[r.clamp_min(0)][:, None, :, :], box, periodic)
                    near = ((d * d).sum(-1) <= RC * RC) & (p >= 0)[:, :, None] & (r >= 0)[:, None, :]
                    if (dz, dy, dx) == (0, 0, 0):
                        near &= p[:, :, None] < r[:, None, :]
                    t, u, v = torch.nonzero(near, as_tuple=True)
                    out.append(torch.stack([p[t, u], r[t, v]]))
    return torch.cat(out, 1)


class _System:
    """Pairs with i a Pd site where the two differ, and each type's chunks."""

    def __init__(self, p):
        dev = "cuda"
        X = torch.from_numpy(np.ascontiguousarray(p["X"])).to(dev).reshape(-1, 4)
        self.p, self.nPd, self.N = p, p["nPd"], len(X)
        self.q, self.u = X[:, :3].contiguous(), math.sqrt(6.0) * X[:, 3]
        self.sigma = X[:, 3]
        self.occ = torch.cat([torch.ones(p["nPd"], dtype=torch.float64, device=dev),
                              torch.from_numpy(np.ascontiguousarray(p["xH"])).to(dev)])
        ij = _pair_list(self.q, p["box"], p["periodic"])
        i, j = torch.minimum(ij[0], ij[1]), torch.maximum(ij[0], ij[1])
        kind = (i >= self.nPd).long() + (j >= self.nPd).long()  # 0 Pd-Pd, 1 Pd-H, 2 H-H
        self.pairs = [(i[kind == t], j[kind == t]) for t in range(3)]

    def chunks(self, t, size=400_000):
        i, j = self.pairs[t]
        for a in range(0, len(i), size):
            yield i[a:a + size], j[a:a + size]

    def radii(self, i, j):
        """Base vector D and the 12 radii: +-u_i on each axis, then -+u_j."""
        D = _wrap(self.q[i] - self.q[j], self.p["box"], self.p["periodic"])
        D2 = (D * D).sum(-1, keepdim=True)
        ui, uj = self.u[i, None], self.u[j, None]
        s2 = torch.cat([D2 + ui * ui + 2 * D * ui, D2 + ui * ui - 2 * D * ui,
                        D2 + uj * uj - 2 * D * uj, D2 + uj * uj + 2 * D * uj], -1)
        return D, torch.sqrt(s2)

    def densities(self):
        f = ((_f_pd, _f_pd), (_f_pd, _f_h), (_f_h, _f_h))
        rho = torch.zeros(self.N, dtype=torch.float64, device=self.q.device)
        for t in range(3):
            for i, j in self.chunks(t):
                _, s = self.radii(i, j)
                # a site's density holds its neighbors' functions: i feels j's
                fi, fj = f[t][0](s).sum(-1), f[t][1](s).sum(-1)
                rho.index_add_(0, i, W * self.occ[j] * fj)
                rho.index_add_(0, j, W * self.occ[i] * fi)
        r = rho.clone().requires_grad_(True)
        F = torch.cat([_embed_pd(r[:self.nPd]), _embed_h(r[self.nPd:])])
        dF, = torch.autograd.grad(F.sum(), r)
        return rho, F.detach(), dF


def _objective(p):
    S = _System(p)
    T = p["T"]
    _, F, dF = S.densities()
    V = float((S.occ * F).sum())
    Gq = torch.zeros_like(S.q)
    Gs = torch.zeros_like(S.sigma)
    f = ((_f_pd, _f_pd, _phi_pd), (_f_pd, _f_h, _phi_pdh), (_f_h, _f_h, _phi_h))
    for t in range(3):
        for i, j in S.chunks(t):
            D, s = S.radii(i, j)
            s = s.requires_grad_(True)
            phi = f[t][2](s)
            g = dF[i, None] * f[t][1](s) + dF[j, None] * f[t][0](s) + phi
            c, = torch.autograd.grad(g.sum(), s)
            w = W * S.occ[i] * S.occ[j]
            V += float((w * phi.detach().sum(-1)).sum())
            c = c / s.detach()
            a, b, d, e = c[:, 0:3], c[:, 3:6], c[:, 6:9], c[:, 9:12]
            ui, uj = S.u[i, None], S.u[j, None]
            h = w[:, None] * (D * c.sum(-1, keepdim=True) + ui * (a - b) + uj * (e - d))
            Gq.index_add_(0, i, h)
            Gq.index_add_(0, j, -h)
            Gs.index_add_(0, i, w * (D * (a - b) + ui * (a + b)).sum(-1))
            Gs.index_add_(0, j, w * (D * (e - d) + uj * (e + d)).sum(-1))
    G = torch.cat([Gq / T, (math.sqrt(6.0) / T * Gs - 3.0 * KB * S.occ / S.sigma)[:, None]], 1).reshape(-1)
    return V / T - 3.0 * KB * float((S.occ * torch.log(S.sigma)).sum()), G


def _occupancy(p):
    S = _System(p)
    T, nPd = p["T"], S.nPd
    _, F, dF = S.densities()
    acc = F.clone()
    for i, j in S.chunks(1):
        _, s = S.radii(i, j)
        acc.index_add_(0, j, W * (dF[i, None] * _f_h(s) + _phi_pdh(s)).sum(-1))
    near = []
    for i, j in S.chunks(2):
        D, s = S.radii(i, j)
        fh, ph = _f_h(s).sum(-1), _phi_h(s).sum(-1)
        acc.index_add_(0, i, W * S.occ[j] * (dF[j] * fh + ph))
        acc.index_add_(0, j, W * S.occ[i] * (dF[i] * fh + ph))
        first = (D * D).sum(-1) < 0.75 * A0 * A0
        near.append(torch.stack([i[first], j[first]]))
    x = S.occ[nPd:]
    gamma = torch.log(x / (1.0 - x)) + acc[nPd:] / (KB * T) + 1.5
    gamma = torch.where(gamma > GAMMA_BD, torch.full_like(gamma, GAMMA_BD), gamma)
    bd = torch.from_numpy(p["bd"]).to(x.device).long()
    gamma[bd] = GAMMA_BD
    phi = gamma - torch.log(x / (1.0 - x))
    i, j = torch.cat(near, 1) - nPd
    rate = torch.zeros_like(x)
    for a, b in ((i, j), (j, i)):
        h = (phi[a] - phi[b]) / 2.0
        rate.index_add_(0, a, x[b] * (1 - x[a]) * torch.exp(-h) - x[a] * (1 - x[b]) * torch.exp(h))
    new = torch.clamp(x + NU * math.exp(-QM / (KB * T)) * rate * DT, X_LB, X_UB)
    new[bd] = x[bd]
    inside = torch.ones_like(x, dtype=torch.bool)
    inside[bd] = False
    return {"gamma": gamma, "full": None, "x": new, "mean": float(new.mean()), "interior": float(new[inside].mean())}


def exact(case, seed):
    if case["op"] in ("minimize", "batch"):
        return None  # whole minimizations: a trajectory, not a formula
    p = _inputs(case, seed)
    if case["op"] == "occupancy":
        return _occupancy(p)
    f, G = _objective(p)
    if case["op"] == "eval":
        f = torch.tensor([f], dtype=torch.float64)
    out = {"f": f, "G": G}
    if case["op"] in ("lists", "skin"):
        out["f"] = torch.tensor([f], dtype=torch.float64)
        out.update(most=None, shells=None)
    return out
