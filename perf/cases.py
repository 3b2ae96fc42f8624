"""Workloads of the library's main paths, each through the public entry points of cq_b200.

A case is a dict of plain values.  Its kind says what one pass does:
  product   one block-sparse product (System.mat_mult), either mult type
  lnv_call  the products of one LNV_matrix_multiply call in their data flow: LS = L.S, LH = L.H,
            HLS = LH.S, B = HLS.(LS)^T in the L range, SLS = LS.S, SLSLS = SLS.(LS)^T, LSL = LS.L,
            LSLSL = LSL.(LS)^T in the H range
  batch     many products of independent systems in one call (mat_mult_batch)
  algebra   transposes, sums of equal and of different ranges, traces: what the chain runs between products
  invert    a new geometry: indices of all ranges of the chain, then T = S^-1 (LNV.invert_S)
  solve     a whole density-matrix solve on a resident S and H (LNV.solve), with L and K copied out

Systems are periodic diamond Si cells ("cell": nx x ny x nz conventional cells of 8 atoms) or clusters cut
from the same lattice ("cluster": n atoms), with Gaussian displacements of the case's own (the neighbour lists, and
so the lengths of the matrices, belong to the case; the values come from the seed); blocks are 4 x 4 ("sz"), 13 x 13
("dzp") or both in one system ("mix").  Matrix entries decay with distance as uniform[-1, 1] exp(-r / 3 bohr);
S and H of the chain are the library's synthetic generators.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "conquest-release_b200"))
import cq_b200  # noqa: E402
from cq_b200 import inputs  # noqa: E402

PRECISION = {"fp64": cq_b200.PREC_FP64, "fma": cq_b200.PREC_FP64_FMA, "fp64tc": cq_b200.PREC_FP64_TC,
             "bf16x6": cq_b200.PREC_BF16X6, "bf16x3": cq_b200.PREC_BF16X3}


def listed():
    return [
        # the smallest calls: one product of a 64-atom cell, where launch and call latency count
        dict(name="product_sz64", kind="product", shape="cell", nx=2, ny=2, nz=2, blocks="sz", type=1, ra=8.0, rb=10.0,
             rc=18.0, precision="fp64"),
        # the plain FP64 path's work per LNV call on the 512-atom SZ cell of the headline benchmark
        dict(name="lnv_call_sz512", kind="lnv_call", shape="cell", nx=4, ny=4, nz=4, blocks="sz", rs=10.0, rh=12.0,
             rl=16.0, precision="fp64"),
        # mat_mult C = A.B on the 216-atom DZP cell (A 8, B 12, C 20 bohr)
        dict(name="product_dzp216", kind="product", shape="cell", nx=3, ny=3, nz=3, blocks="dzp", type=1, ra=8.0, rb=12.0,
             rc=20.0, precision="fp64"),
        # a ragged cluster with both block sizes, a product into a shorter range (mult type 2)
        dict(name="product_mix_cluster150_t2", kind="product", shape="cluster", n=150, blocks="mix", type=2, ra=12.0,
             rb=14.0, rc=24.0, precision="fp64"),
        # the plain FP64 path of a DZP request: 64 atoms, the chain's usual ranges
        dict(name="lnv_call_dzp64", kind="lnv_call", shape="cell", nx=2, ny=2, nz=2, blocks="dzp", rs=10.0, rh=12.0,
             rl=16.0, precision="fp64"),
        # the precision form of a DZP request, its FP64 part: FP64 products on the tensor cores
        dict(name="lnv_call_dzp216_fp64tc", kind="lnv_call", shape="cell", nx=3, ny=3, nz=3, blocks="dzp", rs=10.0,
             rh=12.0, rl=16.0, precision="fp64tc"),
        # the precision form of a DZP request, its split phase: three-part bf16 products
        dict(name="lnv_call_dzp216_bf16x6", kind="lnv_call", shape="cell", nx=3, ny=3, nz=3, blocks="dzp", rs=10.0,
             rh=12.0, rl=16.0, precision="bf16x6"),
        # the largest product of the chain (LS.L -> LSL) on 512 DZP atoms with the two-part split
        dict(name="product_dzp512_bf16x3", kind="product", shape="cell", nx=4, ny=4, nz=4, blocks="dzp", type=1, ra=26.0,
             rb=16.0, rc=42.0, precision="bf16x3"),
        # batched solves: one round of products of eight systems of uneven sizes and block types
        dict(name="batch_8_systems", kind="batch", systems=8, nmin=64, nmax=300, seed_set=7, precision="fp64"),
        # the matrix algebra around the products of one LNV call on the 512-atom SZ cell
        dict(name="algebra_sz512", kind="algebra", shape="cell", nx=4, ny=4, nz=4, blocks="sz", rs=10.0, rh=12.0, rl=16.0),
        # a new geometry (an MD step, a served request): index build, pair lists and S^-1
        dict(name="invert_new_sz216", kind="invert", shape="cell", nx=3, ny=3, nz=3, blocks="sz", rs=10.0, rh=12.0,
             rl=16.0, rt=10.0),
        # a whole small solve (a served SZ request): thousands of short products, sums and traces in a row
        dict(name="solve_sz64", kind="solve", shape="cell", nx=2, ny=2, nz=2, blocks="sz", rs=8.0, rh=9.0, rl=10.0,
             rt=8.0, max_outer=1),
    ]


def draw(rng):
    """One more case: the kinds of listed(), cells of 2..4 conventional cells per side, clusters of 20..300
    atoms, ranges between those of the short and the usual truncations, each precision where it is used."""
    kind = rng.choice(["product", "product", "product", "product", "lnv_call", "lnv_call", "lnv_call", "batch", "algebra",
                       "invert", "solve"])
    r1 = lambda a, b: round(rng.uniform(a, b), 2)  # noqa: E731
    if kind == "batch":
        return dict(kind=kind, systems=rng.randint(2, 12), nmin=64, nmax=rng.choice([100, 200, 300]),
                    seed_set=rng.randint(100, 10 ** 6), precision=rng.choice(["fp64", "fp64", "fma"]))
    blocks = rng.choice(["sz", "dzp", "mix"]) if kind in ("product", "lnv_call", "algebra") else "sz"
    big = kind == "product" or blocks == "sz"
    if kind == "solve" or rng.random() < 0.5:
        top = 4 if big and kind not in ("invert", "solve") else 3
        case = dict(kind=kind, shape="cell", nx=rng.randint(2, top), ny=rng.randint(2, top), nz=rng.randint(2, top),
                    blocks=blocks)
    else:
        top = 300 if big else 120
        case = dict(kind=kind, shape="cluster", n=int(round(20 * (top / 20.0) ** rng.random())), blocks=blocks)
    prec = ["fp64", "fp64", "fma"] if blocks == "sz" else ["fp64", "fp64tc", "bf16x6", "bf16x3"]
    if kind == "product":
        t = rng.choice([1, 1, 2])
        ra, rb = r1(6, 16 if blocks != "sz" else 26), r1(6, 16)
        case.update(type=t, ra=ra, rb=rb, rc=round((ra + rb) * (rng.choice([1.0, 0.8]) if t == 1 else 1.0), 2),
                    precision=rng.choice(prec))
    else:
        case.update(rs=r1(6, 10), rh=r1(7, 12), rl=r1(8, 16))
        if kind == "lnv_call":
            case.update(precision=rng.choice(prec))
        if kind in ("invert", "solve"):
            case.update(rt=round(case["rs"], 2))
        if kind == "solve":
            # an untroubled start needs the usual proportions of the ranges
            case.update(rs=8.0, rh=9.0, rt=8.0, rl=r1(9, 11), max_outer=1)
    return case


# ----------------------------------------------------------------------------------------------------
def _geometry(case):
    if case["shape"] == "cell":
        coords, cell = inputs.diamond_si((case["nx"], case["ny"], case["nz"]), sigma=0.1, seed=2)
    else:
        coords, cell = inputs.si_cluster(case["n"], sigma=0.1, seed=2, vacuum=15.0)
    n = len(coords)
    if case["blocks"] == "sz":
        nsf = np.full(n, 4, np.int32)
    elif case["blocks"] == "dzp":
        nsf = np.full(n, 13, np.int32)
    else:
        nsf = np.where(np.arange(n) % 3 == 0, 13, 4).astype(np.int32)
    return coords, cell, nsf


def _sizes(system, r):
    nd_i = np.repeat(system.geti("ndimi", r), system.geti("n_nab", r))
    return nd_i, system.geti("ndimj", r)


def _random(system, r, gen):
    """uniform[-1, 1] exp(-radius / 3) per element of range r, on the GPU."""
    nd_i, nd_j = _sizes(system, r)
    amp = torch.exp(torch.from_numpy(system.radius(r)).cuda() / -3.0)
    u = torch.rand(system.length(r), dtype=torch.float64, device="cuda", generator=gen)
    return (2.0 * u - 1.0) * torch.repeat_interleave(amp, torch.from_numpy(nd_i * nd_j).cuda())


def _empty(system, r):
    return torch.zeros(max(system.length(r), 1), dtype=torch.float64, device="cuda")[:system.length(r)]


def _overlap(system, r, seed):
    """The generator's S with its overlaps weakened by a seeded factor of 0.9 to 1 (the onsite block stays 1)."""
    S, eye = _empty(system, r), _empty(system, r)
    torch.cuda.synchronize()
    system.generate_SH(r, 0, seed, S)
    system.synchronize()
    nsf, first = system.geti("ndimi", r), system.geti("onsite", r) - 1
    eye[torch.from_numpy(np.concatenate([f + np.arange(n) * (n + 1) for f, n in zip(first, nsf)])).cuda()] = 1.0
    f = 0.9 + 0.1 * float(np.random.default_rng(seed).random())
    return f * S + (1.0 - f) * eye


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _call_ranges(case):
    full = cq_b200.lnv_ranges(case["rs"], case["rh"], case["rl"], case.get("rt", case["rs"]))
    return {k: full[k] for k in ("S", "H", "L", "LS", "LH", "LSL", "SLS")}


# the products of one LNV call: (output, mult type, ra, rb, rc, a, b, c) with the roles of mat_mult
_CALL = (("LS", 1, "L", "S", "LS", "L", "S", "LS"), ("LH", 1, "L", "H", "LH", "L", "H", "LH"),
         ("HLS", 1, "LH", "S", "LSL", "LH", "S", "HLS"), ("B", 2, "L", "LS", "LSL", "B", "LS", "HLS"),
         ("SLS", 1, "LS", "S", "SLS", "LS", "S", "SLS"), ("SLSLS", 2, "L", "LS", "SLS", "SLSLS", "LS", "SLS"),
         ("LSL", 1, "LS", "L", "LSL", "LS", "L", "LSL"), ("LSLSL", 2, "H", "LS", "LSL", "LSLSL", "LS", "LSL"))
_RANGE_OF = {"L": "L", "S": "S", "H": "H", "LS": "LS", "LH": "LH", "HLS": "LSL", "B": "L", "SLS": "SLS", "SLSLS": "L",
             "LSL": "LSL", "LSLSL": "H"}


def _batch_items(case):
    """The systems of a batch: sizes log-uniform, cells and clusters, block types and mult types in turn; both
    the mixed-size products and the 4 x 4 ones travel in one call."""
    rs = np.random.default_rng(case["seed_set"])
    items = []
    for k in range(case["systems"]):
        n = int(round(np.exp(rs.uniform(np.log(case["nmin"]), np.log(case["nmax"])))))
        blocks = ("sz", "dzp", "sz", "mix")[k % 4]
        if blocks != "sz":
            n = min(n, 150)
        sub = dict(shape="cluster", n=n, blocks=blocks)
        if k % 2 == 1:
            m = max(2, int(round((n / 8.0) ** (1.0 / 3.0))))
            sub = dict(shape="cell", nx=m, ny=2, nz=m, blocks=blocks)
        items.append((sub, 1 + (k // 2) % 2))
    return items


_BATCH_RANGES = [10.0, 12.0, 22.0]


def prepare(case, seed):
    kind = case["kind"]
    gen = _generator(seed)
    if kind == "batch":
        state = dict(kind=kind, products=[], outputs=[])
        for sub, t in _batch_items(case):
            s = cq_b200.System(*_geometry(sub), _BATCH_RANGES)
            b = _random(s, 1, gen)
            a, c = (_random(s, 0, gen), _empty(s, 2)) if t == 1 else (_empty(s, 0), _random(s, 2, gen))
            state["products"].append((s, t, 0, 1, 2, a, b, c, PRECISION[case["precision"]]))
            state["outputs"].append(c if t == 1 else a)
        torch.cuda.synchronize()
        return state
    coords, cell, nsf = _geometry(case)
    if kind == "product":
        s = cq_b200.System(coords, cell, nsf, [case["ra"], case["rb"], case["rc"]])
        b = _random(s, 1, gen)
        a, c = (_random(s, 0, gen), _empty(s, 2)) if case["type"] == 1 else (_empty(s, 0), _random(s, 2, gen))
        torch.cuda.synchronize()
        return dict(kind=kind, system=s, type=case["type"], a=a, b=b, c=c, precision=PRECISION[case["precision"]])
    if kind in ("lnv_call", "algebra"):
        rng = _call_ranges(case)
        idx = {k: i for i, k in enumerate(rng)}
        s = cq_b200.System(coords, cell, nsf, list(rng.values()))
        m = {"L": _random(s, idx["L"], gen)}
        if kind == "lnv_call":
            m["S"], m["H"] = _overlap(s, idx["S"], seed), _empty(s, idx["H"])
            torch.cuda.synchronize()
            s.generate_SH(idx["H"], 1, seed, m["H"])
            for name, *_ in _CALL:
                m[name] = _empty(s, idx[_RANGE_OF[name]])
        else:
            for name, r in (("LS", "LS"), ("LSL", "LSL"), ("L2", "L"), ("H", "H")):
                m[name] = _random(s, idx[r], gen)
            for name, r in (("SL", "LS"), ("LT", "L"), ("SLH", "LSL"), ("M", "L"), ("A", "LSL"), ("K", "H")):
                m[name] = _empty(s, idx[r])
        torch.cuda.synchronize()
        return dict(kind=kind, system=s, idx=idx, m=m, precision=PRECISION[case.get("precision", "fp64")])
    if kind == "invert":
        rng = cq_b200.lnv_ranges(case["rs"], case["rh"], case["rl"], case["rt"])
        s = cq_b200.System(coords, cell, nsf, [rng["S"], rng["H"]])
        S, H = _overlap(s, 0, seed), _empty(s, 1)
        torch.cuda.synchronize()
        s.generate_SH(1, 1, seed, H)
        s.synchronize()
        s.close()
        return dict(kind=kind, coords=coords, cell=cell, nsf=nsf, ranges=rng, S=S, H=H, ne=float(len(coords)))
    rng = cq_b200.lnv_ranges(case["rs"], case["rh"], case["rl"], case["rt"])
    idx = {k: i for i, k in enumerate(rng)}
    s = cq_b200.System(coords, cell, nsf, list(rng.values()))
    S, H = _overlap(s, idx["S"], seed), _empty(s, idx["H"])
    torch.cuda.synchronize()
    s.generate_SH(idx["H"], 1, seed, H)
    solver = cq_b200.LNV(s, idx, float(len(coords)), max_outer=case["max_outer"])
    solver.set_SH(S, H)
    s.synchronize()
    return dict(kind=kind, system=s, solver=solver)


def run(state):
    kind = state["kind"]
    if kind == "product":
        state["system"].mat_mult(state["type"], 0, 1, 2, state["a"], state["b"], state["c"], precision=state["precision"])
        return state["c"] if state["type"] == 1 else state["a"]
    if kind == "batch":
        cq_b200.mat_mult_batch(state["products"])
        return state["outputs"]
    if kind == "lnv_call":
        s, idx, m = state["system"], state["idx"], state["m"]
        for _, t, ra, rb, rc, a, b, c in _CALL:
            s.mat_mult(t, idx[ra], idx[rb], idx[rc], m[a], m[b], m[c], precision=state["precision"])
        return {name: m[name] for name, *_ in _CALL}
    if kind == "algebra":
        s, idx, m = state["system"], state["idx"], state["m"]
        s.transpose(idx["LS"], m["LS"], m["SL"])
        s.transpose(idx["LSL"], m["LSL"], m["SLH"])
        s.matrix_sum(idx["LSL"], m["A"], 0.0, idx["LSL"], m["LSL"], 2.0)
        s.matrix_sum(idx["LSL"], m["A"], 1.0, idx["LSL"], m["SLH"], 1.0)
        s.matrix_sum(idx["H"], m["K"], 0.0, idx["LSL"], m["LSL"], 3.0)
        s.matrix_sum(idx["H"], m["K"], 1.0, idx["H"], m["H"], -2.0)
        s.matrix_sum(idx["L"], m["M"], 0.0, idx["LSL"], m["SLH"], 3.0)
        s.matrix_sum(idx["L"], m["M"], 1.0, idx["L"], m["L2"], -1.0)
        s.transpose(idx["L"], m["M"], m["LT"])
        e = s.product_trace(idx["H"], m["H"], m["K"])
        n = s.product_trace(idx["L"], m["L"], m["LT"])
        t = s.trace(idx["L"], m["L"])
        return {"SL": m["SL"], "SLH": m["SLH"], "A": m["A"], "K": m["K"], "M": m["M"], "LT": m["LT"], "traces": [e, n, t]}
    if kind == "invert":
        rng = state["ranges"]
        idx = {k: i for i, k in enumerate(rng)}
        s = cq_b200.System(state["coords"], state["cell"], state["nsf"], list(rng.values()))
        solver = cq_b200.LNV(s, idx, state["ne"])
        solver.set_SH(state["S"], state["H"])
        omega = solver.invert_S()
        T = solver.get("T")
        solver.close()
        s.close()
        return {"omega": omega, "T": T}
    r = state["solver"].solve()
    return {"energy": r["energy"], "electrons": r["electrons"], "products": r["n_products"], "L": state["solver"].get("L"),
            "K": state["solver"].get("K")}


# ----------------------------------------------------------------------------------------------------
def work(case):
    """Bytes: each operand once, each result once.  Flops: 2 nd_i nd_j nd_k per block triple with a stored
    result, one per element of a sum and two per element of a product trace."""
    kind = case["kind"]
    if kind == "batch":
        bytes_, flops = 0, 0
        for sub, t in _batch_items(case):
            s = cq_b200.System(*_geometry(sub), _BATCH_RANGES)
            bytes_ += 8 * sum(s.length(r) for r in range(3))
            flops += s.product_work(t, 0, 1, 2)[1]
        return {"bytes": bytes_, "flops": flops}
    coords, cell, nsf = _geometry(case)
    if kind == "product":
        s = cq_b200.System(coords, cell, nsf, [case["ra"], case["rb"], case["rc"]])
        return {"bytes": 8 * sum(s.length(r) for r in range(3)), "flops": s.product_work(case["type"], 0, 1, 2)[1]}
    if kind in ("lnv_call", "algebra"):
        rng = _call_ranges(case)
        idx = {k: i for i, k in enumerate(rng)}
        s = cq_b200.System(coords, cell, nsf, list(rng.values()))
        n = {k: s.length(i) for k, i in idx.items()}
        if kind == "lnv_call":
            outs = sum(n[_RANGE_OF[o]] for o, *_ in _CALL)
            return {"bytes": 8 * (n["L"] + n["S"] + n["H"] + outs),
                    "flops": sum(s.product_work(t, idx[ra], idx[rb], idx[rc])[1] for _, t, ra, rb, rc, *_ in _CALL)}
        # inputs LS, LSL, L, L2, H; results SL, SLH, A, K, M, LT
        return {"bytes": 8 * (2 * n["LS"] + 3 * n["LSL"] + 4 * n["L"] + 2 * n["H"]),
                "flops": 2 * (n["LSL"] + n["H"] + n["L"]) + 2 * (n["H"] + n["L"])}
    rng = cq_b200.lnv_ranges(case["rs"], case["rh"], case["rl"], case["rt"])
    idx = {k: i for i, k in enumerate(rng)}
    s = cq_b200.System(coords, cell, nsf, list(rng.values()))
    if kind == "invert":
        # about eight Hotelling sweeps of two products each
        f = s.product_work(1, idx["T"], idx["S"], idx["TS"])[1] + s.product_work(2, idx["T"], idx["T"], idx["TS"])[1]
        return {"bytes": 8 * (s.length(idx["S"]) + s.length(idx["T"])), "flops": 8 * f}
    S, H = _overlap(s, idx["S"], 1), _empty(s, idx["H"])
    torch.cuda.synchronize()
    s.generate_SH(idx["H"], 1, 1, H)
    solver = cq_b200.LNV(s, idx, float(len(coords)), max_outer=case["max_outer"])
    solver.set_SH(S, H)
    flops = solver.solve()["flops"]
    return {"bytes": 8 * (s.length(idx["S"]) + 2 * s.length(idx["H"]) + s.length(idx["L"])), "flops": flops}


def tolerance(case):
    """Plain FP64 keeps the bits of the reference's default kernel, and the traces are exact sums: "exact".
    The other precisions: about four times the distance to the 64-bit result, largest over the chain."""
    prec = case.get("precision", "fp64")
    if prec == "fp64":
        return "exact"
    return {"fma": {"rel": 1e-14}, "fp64tc": {"rel": 3e-14}, "bf16x6": {"rel": 6e-7}, "bf16x3": {"rel": 6e-5}}[prec]


# ---------------------------------------------------------------------------------------------------- 64 bits
# Plain torch: the block triples of a product by matching (row atom, column atom, periodic image) keys, no halo,
# partition or pair list.  Only the layout of the matrices (which block lies where) is the library's.
class _Layout:
    def __init__(self, system, r, coords, cell):
        bl = system.blocklist(r, coords, cell)
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.int64)).cuda()  # noqa: E731
        self.i, self.j, self.shift, self.off = dev(bl.ig_i), dev(bl.ig_j), dev(bl.shift), dev(bl.elem_off)
        self.ndi, self.ndj, self.length = dev(bl.nd_i), dev(bl.nd_j), bl.length
        self.n, self.nd = len(coords), int(max(bl.nd_i.max(), bl.nd_j.max())) if len(bl.nd_i) else 1
        self.order = torch.argsort(self.key(self.i, self.j, self.shift))
        self.keys = self.key(self.i, self.j, self.shift)[self.order]
        byrow = torch.argsort(self.i, stable=True)
        self.byrow = byrow
        self.count = torch.bincount(self.i, minlength=self.n)
        self.start = torch.cumsum(self.count, 0) - self.count
        # element (row of the stored nd_j x nd_i view, its column) of every block in an nd x nd padded tile
        g = torch.arange(self.nd, device="cuda")
        self.grid_j, self.grid_i = g[:, None], g[None, :]

    def key(self, i, j, s):
        s = s + 64
        return (((i * self.n + j) * 128 + s[:, 0]) * 128 + s[:, 1]) * 128 + s[:, 2]

    def find(self, i, j, s):
        """Block with this key, or -1."""
        k = self.key(i, j, s)
        p = torch.searchsorted(self.keys, k).clamp(max=max(len(self.keys) - 1, 0))
        return torch.where(self.keys[p] == k, self.order[p], torch.full_like(p, -1))

    def _where(self, q):
        ok = (self.grid_j < self.ndj[q][:, None, None]) & (self.grid_i < self.ndi[q][:, None, None])
        at = self.off[q][:, None, None] + self.grid_j * self.ndi[q][:, None, None] + self.grid_i
        return torch.where(ok, at, torch.zeros_like(at)), ok

    def tiles(self, v, q=None):
        """Blocks q of the values v as padded nd x nd tiles, tile[jj, ii] = block(ii, jj)."""
        q = torch.arange(len(self.i), device="cuda") if q is None else q
        at, ok = self._where(q)
        return torch.where(ok, v[at], torch.zeros((), dtype=v.dtype, device="cuda"))

    def flat(self, tiles):
        out = torch.zeros(self.length, dtype=torch.float64, device="cuda")
        step = 1 << 18
        for q0 in range(0, len(self.i), step):
            q = torch.arange(q0, min(q0 + step, len(self.i)), device="cuda")
            at, ok = self._where(q)
            out[at[ok]] = tiles[q][ok]
        return out


def _exact_product(t, A, B, C, a, b, c):
    """Type 1: C = A.B on C's blocks; type 2: A = C.B^T on A's blocks (64-bit torch)."""
    out, x = (C, A) if t == 1 else (A, C)
    xt, bt = x.tiles(a if t == 1 else c), B.tiles(b)
    acc = torch.zeros(len(out.i), out.nd, out.nd, dtype=torch.float64, device="cuda")
    walk = A                             # blocks (i, k, s); the second operand's row k follows
    step = max(1, (24 << 20) // (out.nd * out.nd * max(1, int(B.count.max()))))
    for q0 in range(0, len(walk.i), step):
        q = torch.arange(q0, min(q0 + step, len(walk.i)), device="cuda")
        k = walk.j[q]
        cnt = B.count[k]
        qq = torch.repeat_interleave(q, cnt)
        first = torch.repeat_interleave(B.start[k] - (torch.cumsum(cnt, 0) - cnt), cnt)
        e = B.byrow[first + torch.arange(len(qq), device="cuda")]
        hit = C.find(walk.i[qq], B.j[e], walk.shift[qq] + B.shift[e])
        keep = hit >= 0
        qq, e, hit = qq[keep], e[keep], hit[keep]
        if t == 1:
            acc.index_add_(0, hit, torch.bmm(bt[e], xt[qq]))
        else:
            acc.index_add_(0, qq, torch.bmm(bt[e].transpose(1, 2), xt[hit]))
    return out.flat(acc)


def _exact_transpose(R, a):
    dest = R.find(R.j, R.i, -R.shift)
    t = R.tiles(a)
    out = torch.zeros_like(t)
    out[dest] = t.transpose(1, 2)
    return R.flat(out)


def _exact_add(A, a, alpha, B, b, beta):
    p = B.find(A.i, A.j, A.shift)
    t = A.tiles(a)
    has = p >= 0
    t[has] = alpha * t[has] + beta * B.tiles(b, p[has])
    return A.flat(t)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("invert", "solve"):
        return None                      # iterations on truncated ranges: no value but their own
    state = prepare(case, seed)
    if kind == "batch":
        outs = []
        for (sub, t), p in zip(_batch_items(case), state["products"]):
            coords, cell, _ = _geometry(sub)
            lay = [_Layout(p[0], r, coords, cell) for r in range(3)]
            outs.append(_exact_product(t, *lay, p[5], p[6], p[7]))
        return outs
    coords, cell, _ = _geometry(case)
    if kind == "product":
        lay = [_Layout(state["system"], r, coords, cell) for r in range(3)]
        return _exact_product(case["type"], *lay, state["a"], state["b"], state["c"])
    idx, m = state["idx"], state["m"]
    lay = {k: _Layout(state["system"], i, coords, cell) for k, i in idx.items()}
    if kind == "lnv_call":
        for name, t, ra, rb, rc, a, b, c in _CALL:
            m[name] = _exact_product(t, lay[ra], lay[rb], lay[rc], m[a], m[b], m[c])
        return {name: m[name] for name, *_ in _CALL}
    SL, SLH = _exact_transpose(lay["LS"], m["LS"]), _exact_transpose(lay["LSL"], m["LSL"])
    A = 2.0 * m["LSL"] + SLH
    K = _exact_add(lay["H"], m["K"], 0.0, lay["LSL"], m["LSL"], 3.0) - 2.0 * m["H"]
    M = _exact_add(lay["L"], m["M"], 0.0, lay["LSL"], SLH, 3.0) - m["L2"]
    LT = _exact_transpose(lay["L"], M)
    on = (lay["L"].i == lay["L"].j) & (lay["L"].shift == 0).all(1)
    tr = torch.diagonal(lay["L"].tiles(m["L"], on.nonzero()[:, 0]), dim1=1, dim2=2).sum()
    return {"SL": SL, "SLH": SLH, "A": A, "K": K, "M": M, "LT": LT,
            "traces": [float((m["H"] * K).sum()), float((m["L"] * LT).sum()), float(tr)]}
