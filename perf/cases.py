"""Timed cases of the residual/update path: what a user of this framework has it do, small to large.

Five uses, each through the public Python API (euler3d_b200.api):

* ``iterate``   restart from a checkpoint, run outer iterations with the fused kernels, write the
                checkpoint back (e3d_state_import / e3d_iterate / e3d_state_export); FP64 is the
                drop-in arithmetic, FP32 the bulk variant; tetrahedra in one or more blocks, or
                hexahedra; first or second order; with or without residual smoothing
* ``strategy``  the same through the strategy objects, method by method, as a program that keeps the
                reference's call sequence does
* ``batch``     a Mach/alpha sweep on meshes of uneven size advanced together (e3d_batch_solve)
* ``finish``    the phase of a sweep below the FP32 floor: batch iterations in difference form
* ``train`` / ``warm``  training steps of the warm-start network, and a warm start with it

``listed`` are the sizes the configurations, tests and benchmark of this repository use, from a
fixture-sized mesh to the 3.07M-tetrahedron workload; ``draw`` spreads over the same ranges.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from euler3d_b200 import api, meshgen
from euler3d_b200 import sweep

GAMMA = 1.4
ORDER = "none+boundary_last"  # the library's default device order of a block's cells
WARM_DATA = os.path.join(os.path.dirname(os.path.abspath(sweep.__file__)), "data", "warmstart_channel_ausm1.npz")


def _flow(name, mesh, n, blocks, precision, order, flux, iters, gradient="leastsquares", limiter="venkatakrishnan",
          mach=0.5, aoa=0.0, nz=1, smoothing=0, kind="iterate"):
    return dict(name=name, kind=kind, mesh=mesh, n=n, nz=nz, blocks=blocks, precision=precision, order=order, flux=flux,
                gradient=gradient, limiter=limiter, mach=mach, aoa=aoa, smoothing=smoothing, iters=iters)


def listed():
    return [
        # a unit-test-sized mesh (the fixtures' order of size): launch latency decides
        _flow("fixture_1k_fp64", "bump", 6, 1, "fp64", 1, "roe", 20),
        # the plain configuration: 20^3 x 6 tetrahedra, first-order Roe, drop-in FP64
        _flow("plain_48k_fp64", "bump", 20, 1, "fp64", 1, "roe", 50),
        # a hexahedron mesh with symmetry planes (the marker mix of a NACA section mesh), Green-Gauss
        _flow("hex_65k_fp64", "hex", 64, 1, "fp64", 2, "ausm", 20, "greengauss", "barthjespersen", 0.6, 1.25, nz=16),
        # second order on several blocks in the drop-in arithmetic
        _flow("second_order_663k_fp64", "bump", 48, 4, "fp64", 2, "roe", 10, mach=0.7, aoa=1.25),
        # the wing's scheme (AUSM + least squares + Venkatakrishnan) on an ordinary odd-sized mesh, FP32
        _flow("ausm_304k_fp32", "bump", 37, 1, "fp32", 2, "ausm", 20, mach=0.8, aoa=3.0),
        # the second-order workload the benchmark quotes: 3.07M tetrahedra in 16 blocks, FP32
        _flow("second_order_3m_fp32", "bump", 80, 16, "fp32", 2, "roe", 20, mach=0.7, aoa=1.25),
        # the drop-in adapters: the reference's own call sequence, block after block
        _flow("strategy_82k_fp64", "bump", 24, 2, "fp64", 2, "roe", 2, mach=0.7, aoa=1.25, kind="strategy"),
        # residual smoothing (a deck option of the reference), Green-Gauss + Barth-Jespersen + AUSM
        _flow("smoothed_25k_fp64", "bump", 16, 1, "fp64", 2, "ausm", 8, "greengauss", "barthjespersen", 0.6, 2.0,
              smoothing=1),
        # a polar sweep: uneven meshes advanced together, second order, FP32
        dict(name="sweep_batch_fp32", kind="batch", sizes="25,14,31,19,22,28", sides="farfield", precision="fp32", order=2,
             flux="ausm", gradient="greengauss", limiter="barthjespersen", iters=40),
        # the finishing phase of the warm-start sweep: first-order AUSM channels in difference form
        dict(name="sweep_finish", kind="finish", sizes="25,18,29", sides="channel", precision="fp32", order=1, flux="ausm",
             gradient="leastsquares", limiter="venkatakrishnan", start=100, iters=100),
        # minibatch training of the warm-start network at the API's default batch
        dict(name="train_16k", kind="train", samples=200000, batch=16384, steps=10),
        # a warm start of one case: features of every cell, the network, the state written
        dict(name="warm_start_384k", kind="warm", n=40, blocks=1, mach=0.55, aoa=2.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, n):
    return rng.choice([b for b in (1, 1, 2, 3, 4, 5, 8) if n % b == 0 and n // b >= 2])


def draw(rng):
    kind = rng.choice(["iterate"] * 9 + ["strategy", "batch", "batch", "finish", "train", "train", "warm", "warm"])
    mach, aoa = round(rng.uniform(0.3, 0.8), 3), round(rng.uniform(-2.0, 6.0), 3)
    if kind in ("iterate", "strategy"):
        hexes = rng.random() < 0.25
        n = _log_int(rng, 5, 40 if kind == "strategy" else 64)
        nz = rng.randint(1, max(1, n // 2)) if hexes else 1
        cells = n * n * nz if hexes else 6 * n ** 3
        order = rng.choice([1, 2, 2])
        smoothing = 1 if kind == "iterate" and rng.random() < 0.15 else 0
        precision = "fp64" if kind == "strategy" or smoothing else rng.choice(["fp64", "fp32"])
        iters = max(4, min(40, 3000000 // cells)) if kind == "iterate" else 2
        c = _flow("", "hex" if hexes else "bump", n, 1 if hexes else _split(rng, n), precision, order,
                  rng.choice(["roe", "ausm"]), iters, rng.choice(["leastsquares", "greengauss"]),
                  rng.choice(["venkatakrishnan", "barthjespersen"]), mach, aoa, nz, smoothing, kind)
        del c["name"]
        return c
    if kind in ("batch", "finish"):
        sizes = ",".join(str(rng.randint(8, 32)) for _ in range(rng.randint(2, 6)))
        if kind == "finish":
            return dict(kind=kind, sizes=sizes, sides="channel", precision="fp32", order=1, flux="ausm",
                        gradient="leastsquares", limiter="venkatakrishnan", start=100, iters=rng.choice([50, 100]))
        return dict(kind=kind, sizes=sizes, sides=rng.choice(["farfield", "channel"]), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    order=rng.choice([1, 2]), flux="ausm", gradient="greengauss", limiter="barthjespersen",
                    iters=rng.randint(20, 60))
    if kind == "train":
        return dict(kind=kind, samples=_log_int(rng, 5000, 400000), batch=_log_int(rng, 1024, 65536), steps=rng.randint(4, 12))
    n = _log_int(rng, 8, 56)
    return dict(kind=kind, n=n, blocks=_split(rng, n), mach=mach, aoa=aoa)


# ------------------------------------------------------------------ inputs
_cases = {}  # host meshes of this process, as a program that runs several states on one mesh keeps them


def _deck(c, mach, aoa):
    return meshgen.Deck(topology="", mach=mach, aoa_deg=aoa, max_iter=10 ** 9, criterion=-50.0, flux=c.get("flux", "ausm"),
                        order=c.get("order", 1), gradient=c.get("gradient", "leastsquares"),
                        limiter=c.get("limiter", "venkatakrishnan"), smoothing=c.get("smoothing", 0))


def _load(c, mesh, n, nz, blocks, sides, mach, aoa):
    d = _deck(c, mach, aoa)
    key = (mesh, n, nz, blocks, sides, mach, aoa, d.flux, d.order, d.gradient, d.limiter, d.smoothing)
    if key not in _cases:
        with tempfile.TemporaryDirectory() as td:
            if mesh == "hex":
                path = meshgen.write_hex_case(td, n, nz, deck=d)
            else:
                path = meshgen.write_case(td, n, blocks, deck=d, sides=sides)
            _cases[key] = api.Case(path)
    return _cases[key]


def _sweep_cases(c):
    """The sweep's meshes with Mach and alpha spread over their ranges, one of each per mesh."""
    sizes = [int(x) for x in c["sizes"].split(",")]
    out = []
    for i, n in enumerate(sizes):
        t = (i + 0.5) / len(sizes)
        out.append(_load(c, "bump", n, 1, 1, c["sides"], round(0.3 + 0.5 * t, 3), round(6.0 - 8.0 * t, 3)))
    return out


def _freestream(deck):
    a, q = math.radians(deck.aoa_deg), deck.mach * math.sqrt(deck.gamma)
    return np.array([1.0, q * math.cos(a), q * math.sin(a), 0.0, 1.0])


def _field(case, b, seed, single):
    """A smooth disturbed flow at the cell centres of one block, [5][n_all]: freestream and a few waves."""
    x = case.get(b, "cell_center").reshape(-1, 3)
    rng = np.random.default_rng([seed, 77])
    free = _freestream(case.deck)
    q = np.empty((5, x.shape[0]))
    for v in range(5):
        k, ph = rng.uniform(1.0, 5.0, (3, 3)), rng.uniform(0, 2 * math.pi, 3)
        wave = sum(np.sin(x @ k[i] + ph[i]) for i in range(3)) / 3
        q[v] = free[v] + 0.04 * wave
    return q.astype(np.float32).astype(np.float64) if single else q


def _conservative(q):
    return np.stack([q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3],
                     0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) + q[4] / (GAMMA - 1.0)])


def _fill(solver, cases, seed):
    b = 0
    for i, case in enumerate(cases):
        for k in range(case.n_blocks):
            q = _field(case, k, seed + 1000 * i, solver.precision == "fp32")
            solver.set(b, "prim", q.ravel())
            if solver.precision == "fp32":  # the FP32 variant carries W in FP64
                solver.set(b, "w0", _conservative(q[:, :case.block_info(k).n_real]).ravel())
            b += 1
    api.halo(solver)


def _pinned(n):
    return torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()


def _flow_case(c):
    return _load(c, c["mesh"], c["n"], c["nz"], c["blocks"], "farfield", c["mach"], c["aoa"])


def _samples(c, seed):
    """Training rows: features in the channel's ranges and a smooth state near each row's freestream."""
    rng = np.random.default_rng([seed, 5])
    n = c["samples"]
    f = np.column_stack([rng.uniform(0, 1, (n, 3)), rng.uniform(0, 0.9, n), rng.uniform(0.3, 0.8, n),
                         rng.uniform(-2, 6, n)]).astype(np.float32)
    x = f.astype(np.float64)
    a, m = np.radians(x[:, 5]), x[:, 4] * math.sqrt(GAMMA)
    bump = np.exp(-((x[:, 0] - 0.5) ** 2) / 0.04) * np.exp(-3 * x[:, 3]) * x[:, 4]
    r = 1 - 0.2 * bump
    u, v, w = m * np.cos(a) * (1 + 0.1 * bump), m * np.sin(a) + 0.1 * np.sin(6 * x[:, 0]) * bump, 0.02 * np.cos(4 * x[:, 2]) * bump
    p = 1 - 0.25 * bump
    s = np.column_stack([r, r * u, r * v, r * w, 0.5 * r * (u * u + v * v + w * w) + p / (GAMMA - 1)]).astype(np.float32)
    return f, s


def _weights(seed):
    """Initial weights of the network, its flat layout: W b of 16 -> 128 -> 128 -> 128 -> 8 (6 inputs, 5 outputs used)."""
    rng = np.random.default_rng([seed, 9])
    out = []
    for rows, cols, used_rows, used_cols, scale in ((128, 16, 128, 6, 1.0), (128, 128, 128, 128, 1.0),
                                                    (128, 128, 128, 128, 1.0), (8, 128, 5, 128, 0.1)):
        w = np.zeros((rows, cols))
        bound = scale * math.sqrt(6.0 / used_cols)
        w[:used_rows, :used_cols] = rng.uniform(-bound, bound, (used_rows, used_cols))
        out += [w.ravel(), np.zeros(rows)]
    return np.concatenate(out).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("iterate", "strategy"):
        hc = _flow_case(case)
        s = api.Solver(hc, precision=case["precision"])
        _fill(s, [hc], seed)
        nbytes = s.state_bytes()
        start, end = _pinned(nbytes), _pinned(nbytes)
        s.export_state(start)
        return dict(case=case, solver=s, start=start, end=end, reference=api.ReferenceSolver(s) if kind == "strategy" else None)
    if kind in ("batch", "finish"):
        cases = _sweep_cases(case)
        b = api.Batch(cases, precision=case["precision"])
        _fill(b, cases, seed)
        done = 0
        if kind == "finish":  # the FP32 phase comes first
            done = case["start"]
            b.solve_batch(done, -50.0, iters_per_launch=50)
            api.set_precision(b, "fp32-delta")
        return dict(case=case, batch=b, done=done)
    if kind == "train":
        m = api.Surrogate(seed=seed)
        m.set_params(_weights(seed))
        m.add_samples(*_samples(case, seed))
        return dict(case=case, model=m)
    hc = _load(dict(order=1, flux="ausm"), "bump", case["n"], 1, case["blocks"], "channel", case["mach"], case["aoa"])
    s = api.Solver(hc, precision="fp32")
    m, _ = sweep.load_surrogate(WARM_DATA)
    params, _ = m.get_params()  # another seed, another (slightly retrained) network
    m.set_params(params * (1 + 0.01 * np.random.default_rng(seed).standard_normal(params.size)).astype(np.float32))
    s.iterate(1)
    return dict(case=case, solver=s, model=m, end=_pinned(s.state_bytes()))


# ------------------------------------------------------------------ one pass
def _n_cells(case):
    info = [case.block_info(b) for b in range(case.n_blocks)]
    return sum(i.n_real for i in info), sum(i.n_all for i in info)


def _primitives(solver, blob):
    """The checkpoint's primitives of every cell: they come before W0 (five doubles per real cell)."""
    nr, na = _n_cells(solver.case)
    t = np.float32 if solver.precision == "fp32" else np.float64
    size = 5 * na * np.dtype(t).itemsize
    at = blob.size - 40 * nr - size
    return blob[at:at + size].view(t)


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("iterate", "strategy"):
        s = state["solver"]
        s.import_state(state["start"])
        if kind == "iterate":
            s.iterate(c["iters"])
        else:
            flow = state["reference"].iterate(c["iters"])
        s.export_state(state["end"])
        out = {"prim": _primitives(s, state["end"])}
        if kind == "strategy":
            out["flow"] = flow[-1]
        elif s.precision == "fp64":
            out["flow"] = s.flow_data()
        return out
    if kind in ("batch", "finish"):
        b = state["batch"]
        state["done"] += c["iters"]
        b.solve_batch(state["done"], -50.0, iters_per_launch=50)
        prim = [b.get(i, "prim") for i in range(b.n_blocks)]
        # the FP32 variant's primitives are FP32 values
        return [q.astype(np.float32) if c["precision"] == "fp32" else q for q in prim]
    if kind == "train":
        _, loss = state["model"].train(c["steps"], c["batch"])
        params, norm = state["model"].get_params()
        return {"params": params, "norm": norm, "loss": loss}
    n = state["model"].warm_start(state["solver"])
    state["solver"].export_state(state["end"])
    return {"prim": _primitives(state["solver"], state["end"]), "fallback": n}


# ------------------------------------------------------------------ work of one pass
def _flow_work(cells, faces, b, order, stages=5):
    # per stage and cell: the state read and written, W0 read; per face: its two cells, area vector and (second
    # order) the two r-vectors; per iteration: the residual norms' sums and the time step in passing
    by = stages * (cells * (10 * b + 40) + faces * (8 + 3 * b + (6 * b if order == 2 else 0)))
    fl = stages * (faces * (180 + (60 if order == 2 else 0)) + cells * (40 + (200 if order == 2 else 0)))
    return by, fl


def work(case):
    kind = case["kind"]
    if kind in ("iterate", "strategy"):
        hexes = case["mesh"] == "hex"
        n = case["n"]
        cells = n * n * case["nz"] if hexes else 6 * n ** 3
        b = 8 if case["precision"] == "fp64" else 4
        by, fl = _flow_work(cells, (3 if hexes else 2) * cells, b, case["order"])
        return dict(bytes=case["iters"] * by + cells * 2 * (5 * b + 40), flops=case["iters"] * fl)
    if kind in ("batch", "finish"):
        cells = sum(6 * int(x) ** 3 for x in case["sizes"].split(","))
        b = 8 if case["precision"] == "fp64" else 4
        by, fl = _flow_work(cells, 2 * cells, b, case["order"])
        return dict(bytes=case["iters"] * by + cells * 40, flops=case["iters"] * fl)
    weights = 6 * 128 + 2 * 128 * 128 + 5 * 128
    if kind == "train":
        rows = case["steps"] * case["batch"]
        return dict(bytes=rows * 44 + case["steps"] * 36232 * 28, flops=6 * weights * rows)
    cells = 6 * case["n"] ** 3
    return dict(bytes=cells * (12 + 2 * 20 + 40), flops=2 * weights * cells)


# ------------------------------------------------------------------ 64-bit values
class _Plain:
    """The discrete equations on whole arrays in 64 bits: faces scattered to cells with index_add."""

    def __init__(self, case):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        d = self.deck = case.deck
        self.case, self.g = case, d.gamma
        get = lambda b, k: case.get(b, k)  # noqa: E731
        f, off, foff = {}, 0, 0
        add = lambda k, a: f.setdefault(k, []).append(a)  # noqa: E731
        self.real, self.block, self.wall = [], [], []
        conn = []
        for b in range(case.n_blocks):
            info = case.block_info(b)
            fc = get(b, "face_cells").reshape(-1, 2).astype(np.int64)
            add("lr", fc + off)
            for k in ("face_normal", "r_left", "r_right", "face_center"):
                add(k, get(b, k).reshape(-1, 3))
            add("area", get(b, "face_area"))
            add("vol", get(b, "cell_volume"))
            ptr = get(b, "cell_face_ptr")[:info.n_real + 1].astype(np.int64)
            rep = np.repeat(np.arange(info.n_real), np.diff(ptr)) + off
            add("scell", rep)
            add("snbr", get(b, "cell_cells")[:ptr[-1]].astype(np.int64) + off)
            add("lsw", get(b, "ls_weights").reshape(-1, 3)[:ptr[-1]])
            ghost_face = np.full(info.n_all, -1, dtype=np.int64)
            g = fc[:, 1] >= info.n_real
            ghost_face[fc[g, 1]] = np.nonzero(g)[0]
            assert not np.any(fc[:, 0] >= info.n_real)
            kinds, sizes, cells = (get(b, k) for k in ("marker_kind", "marker_size", "marker_cells"))
            kind = np.repeat(kinds, sizes)
            number = np.repeat(np.arange(kinds.size), sizes)
            add("ghost", cells.astype(np.int64) + off)
            add("gface", ghost_face[cells] + foff)
            add("gkind", kind)
            add("grefl", number < info.n_real_boundaries)
            conn.append((kind == 4))
            self.wall.append(torch.as_tensor(get(b, "wall_faces").astype(np.int64) + foff, device=self.dev))
            self.real.append((off, info.n_real, info.n_all))
            off += info.n_all
            foff += fc.shape[0]
        t = {k: torch.as_tensor(np.concatenate(v), device=self.dev) for k, v in f.items()}
        self.__dict__.update(t)
        self.n = off
        self.L, self.R = self.lr[:, 0].contiguous(), self.lr[:, 1].contiguous()
        self.nn = self.face_normal / self.area[:, None]
        self.gin = self.L[self.gface]
        # halo: the two ghosts of one shared face sit at the same face centre
        sel = torch.nonzero(self.gkind == 4).ravel()
        if sel.numel():
            at = torch.round(self.face_center[self.gface[sel]] * 1e6).to(torch.int64)
            key = (at[:, 0] * 2000003 + at[:, 1]) * 2000003 + at[:, 2]
            o = torch.argsort(key)
            a, c = sel[o[0::2]], sel[o[1::2]]
            assert torch.equal(key[o[0::2]], key[o[1::2]])
            self.hdst = torch.cat([self.ghost[a], self.ghost[c]])
            self.hsrc = torch.cat([self.gin[c], self.gin[a]])
        else:
            self.hdst = None
        is_real = torch.zeros(self.n, dtype=torch.bool, device=self.dev)
        for o, nr, _ in self.real:
            is_real[o:o + nr] = True
        self.is_real = is_real
        self.reals = torch.nonzero(is_real).ravel()
        self.slots = torch.zeros(self.n, dtype=torch.float64, device=self.dev).index_add_(
            0, self.scell, torch.ones_like(self.scell, dtype=torch.float64))
        self.free = torch.as_tensor(_freestream(d), device=self.dev)

    def halo(self, q):
        if self.hdst is not None:
            q[self.hdst] = q[self.hsrc]

    def boundary(self, q):
        sel = torch.nonzero(self.grefl & (self.gkind != 4)).ravel()
        gh, n, x = self.ghost[sel], self.nn[self.gface[sel]], q[self.gin[sel]]
        far = (self.gkind[sel] == 2)[:, None]
        un = (x[:, 1:4] * n).sum(1, keepdim=True)
        slip = x.clone()
        slip[:, 1:4] = 2 * (x[:, 1:4] - un * n) - x[:, 1:4]
        r, p, c = x[:, :1], x[:, 4:], torch.sqrt(self.g * x[:, 4:] / x[:, :1])
        fr = self.free[None, :]
        pb = 0.5 * (fr[:, 4:] + p - r * c * (n * (fr[:, 1:4] - x[:, 1:4])).sum(1, keepdim=True))
        inflow = torch.cat([fr[:, :1] + (pb - fr[:, 4:]) / (c * c), fr[:, 1:4] - n * (fr[:, 4:] - pb) / (r * c), pb], 1)
        pe = fr[:, 4:].expand_as(p)
        outflow = torch.cat([r + (pe - p) / (c * c), x[:, 1:4] + n * (p - pe) / (r * c), pe], 1)
        sub = 2 * torch.where(un < 0, inflow, outflow) - x
        sup = torch.where(un < 0, 2 * fr - x, x)
        q[gh] = torch.where(far, torch.where((un / c).abs() > 1, sup, sub), slip)

    def limiter(self, d2, hi, lo, eps2):
        if self.deck.limiter == 1:
            D = torch.where(d2 > 0, hi, lo)
            v = (1 / d2) * ((D * D + eps2) * d2 + 2 * d2 * d2 * D) / (D * D + 2 * d2 * d2 + D * d2 + eps2)
            return torch.where(d2 == 0, torch.ones_like(v), v)
        d2 = torch.copysign(d2.abs() + self.deck.omega, d2)
        v = torch.where(d2 > 0, hi, lo) / d2
        return torch.where(d2 == 0, torch.ones_like(v), v.clamp(max=1.0))

    def face_states(self, q):
        qL, qR = q[self.L], q[self.R]
        if self.deck.order != 2:
            return qL, qR
        grad = torch.zeros(self.n, 3, 5, dtype=torch.float64, device=self.dev)
        if self.deck.gradient == 1:
            grad.index_add_(0, self.scell, self.lsw[:, :, None] * (q[self.snbr] - q[self.scell])[:, None, :])
        else:
            a = self.face_normal[:, :, None] * (0.5 * (qL + qR))[:, None, :]
            grad.index_add_(0, self.L, a)
            grad.index_add_(0, self.R, -a)
            grad /= self.vol[:, None, None]
        n = self.nn[self.gface]
        gi = grad[self.gin]
        grad[self.ghost] = torch.where(self.grefl[:, None, None],
                                       gi - 2 * n[:, :, None] * (gi * n[:, :, None]).sum(1, keepdim=True), torch.zeros_like(gi))
        hi, lo = q.clone(), q.clone()
        for a, b in ((self.L, qR), (self.R, qL)):
            i = a[:, None].expand(-1, 5)
            hi.scatter_reduce_(0, i, b, "amax")
            lo.scatter_reduce_(0, i, b, "amin")
        hi, lo = hi - q, lo - q
        eps2 = (self.deck.k ** 3 * self.vol)[:, None]
        phi = torch.full((self.n, 5), math.inf, dtype=torch.float64, device=self.dev)
        d = []
        for a, r in ((self.L, self.r_left), (self.R, self.r_right)):
            d2 = (grad[a] * r[:, :, None]).sum(1)
            phi.scatter_reduce_(0, a[:, None].expand(-1, 5), self.limiter(d2, hi[a], lo[a], eps2[a]), "amin")
            d.append(d2)
        return qL + phi[self.L] * d[0], qR + phi[self.R] * d[1]

    def fluxes(self, qL, qR):
        g, gr, n, S = self.g, self.g / (self.g - 1), self.nn, self.area[:, None]

        def side(q):
            r, u, p = q[:, :1], q[:, 1:4], q[:, 4:]
            return r, u, p, 0.5 * (u * u).sum(1, keepdim=True) + gr * p / r, (u * n).sum(1, keepdim=True)

        rL, uL, pL, HL, VL = side(qL)
        rR, uR, pR, HR, VR = side(qR)
        if self.deck.flux == 0:
            FL = torch.cat([rL * VL, rL * uL * VL + n * pL, rL * HL * VL], 1)
            FR = torch.cat([rR * VR, rR * uR * VR + n * pR, rR * HR * VR], 1)
            sL, sR = torch.sqrt(rL), torch.sqrt(rR)
            rw, u, H = sL * sR, (uL * sL + uR * sR) / (sL + sR), (HL * sL + HR * sR) / (sL + sR)
            q2, V = (u * u).sum(1, keepdim=True), (u * n).sum(1, keepdim=True)
            c = torch.sqrt((g - 1) * (H - q2 / 2))
            fix = lambda a: torch.where(a <= 0.1 * c, (a * a + 0.01 * c * c) / (0.2 * c), a)  # noqa: E731
            dp, dV, dr, du = pR - pL, VR - VL, rR - rL, uR - uL
            one = torch.ones_like(V)
            k1 = fix((V - c).abs()) * (dp - rw * c * dV) / (2 * c * c)
            k5 = fix((V + c).abs()) * (dp + rw * c * dV) / (2 * c * c)
            k = fix(V.abs())
            e = dr - dp / (c * c)
            D = k1 * torch.cat([one, u - c * n, H - c * V], 1) + k5 * torch.cat([one, u + c * n, H + c * V], 1)
            D = D + k * torch.cat([e, e * u + rw * (du - dV * n), e * q2 / 2 + rw * ((u * du).sum(1, keepdim=True) - V * dV)], 1)
            return 0.5 * (FL + FR) * S, 0.5 * D * S
        cL, cR = torch.sqrt(g * pL / rL), torch.sqrt(g * pR / rR)
        ML, MR = VL / cL, VR / cR
        z = torch.zeros_like(ML)
        Mp = torch.where(ML <= -1, z, torch.where(ML < 1, 0.25 * (ML + 1) ** 2, ML))
        Pp = torch.where(ML <= -1, z, torch.where(ML < 1, pL * 0.25 * (ML + 1) ** 2 * (2 - ML), pL))
        Mm = torch.where(MR <= -1, MR, torch.where(MR < 1, -0.25 * (MR - 1) ** 2, z))
        Pm = torch.where(MR <= -1, pR, torch.where(MR < 1, pR * 0.25 * (1 - MR) ** 2 * (2 + MR), z))
        M, P = Mp + Mm, (Pp + Pm) * S
        FL = rL * cL * torch.cat([torch.ones_like(z), uL, HL], 1)
        FR = rR * cR * torch.cat([torch.ones_like(z), uR, HR], 1)
        F = 0.5 * M * (FL + FR) * S
        F[:, 1:4] += n * P
        a = torch.where(M.abs() > 0.25, M, (M * M + 0.0625) / 0.5).abs()
        return F, 0.5 * a * (FR - FL) * S

    def gather(self, f):
        out = torch.zeros(self.n, 5, dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.L, f).index_add_(0, self.R, -f)

    def smooth(self, R):
        j = R / (1 + 0.8 * self.slots[:, None])
        j[~self.is_real] = 0
        s = torch.zeros_like(R).index_add_(0, self.scell, j[self.snbr])
        return (R + 0.8 * s) / (1 + 0.8 * self.slots[:, None])

    def iterate(self, q, iters):
        alpha, beta = api.RK_TABLES[self.deck.stages]
        rl = self.reals
        rd = torch.zeros(self.n, 5, dtype=torch.float64, device=self.dev)
        for _ in range(iters):
            x = q[rl]
            W0 = torch.cat([x[:, :1], x[:, :1] * x[:, 1:4],
                            0.5 * x[:, :1] * (x[:, 1:4] ** 2).sum(1, keepdim=True) + x[:, 4:] / (self.g - 1)], 1)
            c = torch.sqrt(self.g * q[:, 4] / q[:, 0])
            sr = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
            for a in (self.L, self.R):
                sr.index_add_(0, a, ((q[a, 1:4] * self.nn).sum(1).abs() + c[a]) * self.area)
            dtv = (self.deck.cfl / sr[rl])[:, None]
            for a, b in zip(alpha, beta):
                fc, fd = self.fluxes(*self.face_states(q))
                rc, rd = self.gather(fc), rd * (1 - b) + b * self.gather(fd)
                if self.deck.smoothing:
                    rc, rd = self.smooth(rc), self.smooth(rd)
                W = W0 - a * dtv * (rc - rd)[rl]
                q = q.clone()
                u = W[:, 1:4] / W[:, :1]
                q[rl] = torch.cat([W[:, :1], u, (self.g - 1) * (W[:, 4:] - 0.5 * W[:, :1] * (u * u).sum(1, keepdim=True))], 1)
                self.boundary(q)
            flow = self.flow(q, rc - rd)
            self.halo(q)
        return q, flow

    def flow(self, q, r):
        out = []
        d = self.deck
        for (o, nr, _), w in zip(self.real, self.wall):
            cp = (0.5 * (q[self.L[w], 4] + q[self.R[w], 4]) - 1) / (0.5 * d.gamma * d.mach ** 2 * d.cmac)
            fx, fy, fz = (cp[:, None] * self.face_normal[w]).unbind(1)
            x, y, z = self.face_center[w].unbind(1)
            out.append(torch.cat([(r[o:o + nr] ** 2).sum(0),
                                  torch.stack([t.sum() for t in (fy, fx, y * fz - z * fy, z * fx - x * fz, x * fy - y * fx)])]))
        return torch.stack(out).cpu().numpy()

    def start(self, seed, single):
        q = np.concatenate([_field(self.case, b, seed, single).T for b in range(self.case.n_blocks)])
        q = torch.as_tensor(q, device=self.dev)
        self.halo(q)
        return q

    def device_order(self, q):
        """Packed as the checkpoint has it: all real cells in device order, then all ghosts; (rho, u, v, w), then p."""
        real, ghost = [], []
        for b, (o, nr, na) in enumerate(self.real):
            real.append(o + self.case.cell_order(b, ORDER).astype(np.int64))
            ghost.append(np.arange(o + nr, o + na))
        q = q[torch.as_tensor(np.concatenate(real + ghost), device=self.dev)]
        return torch.cat([q[:, :4].reshape(-1), q[:, 4]]).cpu().numpy()


def _network(params, norm, f):
    """The warm-start network's output in 64 bits on raw features (n x 6): scaled deviations from freestream."""
    H, I = 128, 16
    at = 0

    def take(*shape):
        nonlocal at
        n = int(np.prod(shape))
        at += n
        return params[at - n:at].reshape(*shape)

    W1, b1, W2, b2, W3, b3, W4, b4 = take(H, I), take(H), take(H, H), take(H), take(H, H), take(H), take(8, H), take(8)
    gelu = torch.nn.functional.gelu
    h = gelu(((f - norm[:6]) / norm[8:14]) @ W1[:, :6].T + b1)
    h = gelu(h @ W2.T + b2)
    h = gelu(h @ W3.T + b3)
    return (h @ W4.T + b4)[:, :5]


def _wfree(f):
    a, q = torch.deg2rad(f[:, 5]), f[:, 4] * math.sqrt(GAMMA)
    u, v = q * torch.cos(a), q * torch.sin(a)
    one = torch.ones_like(u)
    return torch.stack([one, u, v, 0 * one, 0.5 * (u * u + v * v) + one / (GAMMA - 1)], 1)


def _mix(x):
    """splitmix64's finaliser, the minibatches' hash."""
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _exact_train(c, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    w = torch.tensor(_weights(seed), dtype=torch.float64, device=dev)
    f, s = (torch.as_tensor(a.astype(np.float64), device=dev) for a in _samples(c, seed))
    dev_t = s - _wfree(f)
    norm = torch.zeros(24, dtype=torch.float64, device=dev)
    norm[:6], norm[8:16], norm[16:24] = f.mean(0), 1e-6, 1e-6
    norm[8:14] = f.std(0, unbiased=False)
    norm[16:21] = dev_t.square().mean(0).sqrt()
    m1, m2, losses = torch.zeros_like(w), torch.zeros_like(w), []
    for k in range(c["steps"]):
        i = np.arange(c["batch"], dtype=np.uint64)
        with np.errstate(over="ignore"):
            row = _mix(np.uint64(seed) ^ _mix(np.uint64(k) * np.uint64(0x100000001B3) + i)) % np.uint64(c["samples"])
        row = torch.as_tensor(row.astype(np.int64), device=dev)
        w = w.detach().requires_grad_()
        y = _network(w, norm, f[row])
        loss = ((y - dev_t[row] / norm[16:21]) ** 2).mean()
        g, = torch.autograd.grad(loss, w)
        losses.append(float(loss.detach()))
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        lr = 2e-3 * (0.05 + 0.475 * (1 + math.cos(math.pi * (k / (c["steps"] - 1) if c["steps"] > 1 else 1.0))))
        w = w.detach() - lr * (m1 / (1 - 0.9 ** (k + 1))) / ((m2 / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": w.cpu().numpy(), "norm": norm.cpu().numpy(), "loss": np.array(losses)}


def _exact_warm(c, seed):
    st = prepare(c, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    case = st["solver"].case
    params, norm = (torch.tensor(a, dtype=torch.float64, device=dev) for a in st["model"].get_params())
    # ghosts keep their state: they are taken from the solver as they are
    st["solver"].export_state(st["end"])
    before = _primitives(st["solver"], st["end"]).astype(np.float64)
    nr, na = _n_cells(case)
    xs = np.concatenate([case.get(b, "cell_center").reshape(-1, 3)[:case.block_info(b).n_real][case.cell_order(b, ORDER)]
                         for b in range(case.n_blocks)])
    walls = np.concatenate([case.get(b, "face_center").reshape(-1, 3)[case.get(b, "wall_faces")] for b in range(case.n_blocks)])
    x, w = torch.as_tensor(xs, device=dev), torch.as_tensor(walls, device=dev)
    dist = torch.cat([torch.cdist(p, w, compute_mode="donot_use_mm_for_euclid_dist").amin(1) for p in x.split(8192)])
    d = case.deck
    f = torch.cat([x, dist[:, None], torch.full_like(x[:, :1], d.mach), torch.full_like(x[:, :1], d.aoa_deg)], 1)
    W = _wfree(f) + norm[16:21] * _network(params, norm, f)
    u = W[:, 1:4] / W[:, :1]
    q = torch.cat([W[:, :1], u, (GAMMA - 1) * (W[:, 4:] - 0.5 * W[:, :1] * (u * u).sum(1, keepdim=True))], 1).cpu().numpy()
    before[:4 * nr], before[4 * na:4 * na + nr] = q[:, :4].ravel(), q[:, 4]
    st["solver"].close()
    st["model"].close()
    return {"prim": before, "fallback": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("iterate", "strategy"):
        p = _Plain(_flow_case(case))
        single = case["precision"] == "fp32"
        q, flow = p.iterate(p.start(seed, single), case["iters"])
        return {"prim": p.device_order(q)} if single else {"prim": p.device_order(q), "flow": flow}
    if kind in ("batch", "finish"):
        out = []
        if kind == "finish" and sum(int(x) for x in case["sizes"].split(",")) > 100:
            return None  # takes longer than is sensible
        for i, hc in enumerate(_sweep_cases(case)):
            p = _Plain(hc)
            q, _ = p.iterate(p.start(seed + 1000 * i, case["precision"] == "fp32"), case.get("start", 0) + case["iters"])
            out.append(q.T.contiguous().reshape(-1).cpu().numpy())
        return out
    return _exact_train(case, seed) if kind == "train" else _exact_warm(case, seed)
