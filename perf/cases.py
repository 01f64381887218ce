"""The calls this framework is used for, as cases to be timed and compared.

Grids are the seeded synthetic transmission grids of ``gpusim2grid_b200.synthetic``: the 118-, 2000-, 6500- and
10000-bus ones that the benchmark and the tests run, and grids of the same recipe at any size between.  Each kind of
case is one public entry point as a program calls it:

  single    ``AcPfGPU.resolve``: one power flow, solved again at a new operating point
  sweep     ``compute()`` of ``ContingencyAnalysisGPU`` / ``InjectionSweepGPU`` / ``ScenarioSweepGPU``, rows in place
            (``host``: the rows go in from host arrays and the voltages come back to the host inside the call)
  multi     ``compute_many``: one batch over several grids
  grad      ``batch_power_flow`` and the gradient of a loss of its voltages with respect to the injections
  predict   ``WarmStartMLP.predict``: the warm-start network's inference
  gradients ``WarmStartMLP.gradients``: its forward and backward pass
"""

import dataclasses
import functools
import math

import numpy as np
import torch

import gpusim2grid_b200 as gs
from gpusim2grid_b200.differentiable import batch_power_flow
from gpusim2grid_b200.synthetic import GRID_SPECS, grid_by_name, injection_scenarios, make_grid, n1_branches
from gpusim2grid_b200.warmstart import LearnedStart, WarmStartMLP

SN = 100.0  # MVA, the grids' base power


# ------------------------------------------------------------------- cases
def listed():
    return [
        # an operator's tool re-solving one small grid at every new measurement: latency of one call
        dict(name="single_118", kind="single", n_bus=118, precision="fp64"),
        # the same on a grid of ordinary size
        dict(name="single_2000", kind="single", n_bus=2000, precision="fp64"),
        # full N-1 of a small grid with the facade's default options (FP64, four Newton steps a row), with the branch
        # loadings a security analysis reads; every branch, so the islanding ones are among the rows
        _sweep("n1_118", 118, "n1", 0, limits=True),
        # full N-1 of an ordinary grid with the default options
        _sweep("n1_2000", 2000, "n1", 0),
        # the same in mixed precision on the shared base factor, rows leaving as they converge
        _sweep("n1_2000_mixed", 2000, "n1", 0, **_FAST),
        # the benchmark's headline call: the same rows started from the trained network's voltages
        _sweep("n1_2000_learned", 2000, "n1", 0, start="learned", **_FAST),
        # injection scenarios on a large grid
        _sweep("injections_6500", 6500, "injection", 2048, **_FAST),
        # injection scenarios with outages, host arrays in and host voltages out: the whole call
        _sweep("scenarios_2000_host", 2000, "scenario", 4096, host=True, **_FAST),
        # rows of small and large grids in one batch
        dict(name="grids_118_to_10000", kind="multi", grids="118,2000,6500,10000", rows=256),
        # gradients of a loss through a batch of power flows (forward FP64 sweep, backward adjoint)
        dict(name="grad_2000", kind="grad", n_bus=2000, rows=256),
        # the warm-start network of the 2000-bus grid: inference on one N-1 sweep's rows, and a training batch
        dict(name="predict_2000", kind="predict", n_in=7196, n_out=3598, hidden=1024, layers=2, rows=2944),
        dict(name="gradients_2000", kind="gradients", n_in=7196, n_out=3598, hidden=1024, layers=2, rows=1024),
    ]


_FAST = dict(precision="mixed", scheduling="continuous", strategy="base_chord", nb_iter=10)


def _sweep(name, n_bus, what, rows, precision="fp64", scheduling="chunked", strategy="refactor_every", nb_iter=4,
           start="base", limits=False, host=False):
    c = dict(kind="sweep", n_bus=n_bus, what=what, rows=rows, precision=precision, scheduling=scheduling,
             strategy=strategy, nb_iter=nb_iter, start=start, limits=limits, host=host)
    return dict(c, name=name) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "sweep", "sweep", "sweep", "sweep", "multi", "grad", "predict", "gradients"])
    if kind == "single":
        return dict(kind=kind, n_bus=_log_int(rng, 40, 6500), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "multi":
        n = [_log_int(rng, 60, 600), _log_int(rng, 600, 2500), _log_int(rng, 2500, 8000)]
        return dict(kind=kind, grids=",".join(map(str, n)), rows=_log_int(rng, 16, 300))
    if kind == "grad":
        n = _log_int(rng, 60, 3000)
        return dict(kind=kind, n_bus=n, rows=_log_int(rng, 8, min(2000, 256 * (2000 / n) ** 1.5)))
    if kind in ("predict", "gradients"):
        dim = _log_int(rng, 150, 3598)
        c = dict(kind=kind, n_in=2 * dim, n_out=dim, hidden=rng.choice([256, 512, 1000, 1024]),
                 layers=rng.choice([1, 2, 2, 3]))
        return dict(c, rows=_log_int(rng, 100, 12000) if kind == "predict" else 128 * _log_int(rng, 1, 16))
    what = rng.choice(["n1", "injection", "scenario"])
    if rng.random() < 0.4:  # a factorization per row and step
        n = _log_int(rng, 60, 2500)
        rows = _log_int(rng, 30, min(4000, 2500 * (2000 / n) ** 1.2))
        opts = dict(precision=rng.choice(["fp64", "fp64", "mixed"]), nb_iter=4)
        if rng.random() < 0.4:
            opts.update(scheduling="continuous", nb_iter=10, strategy=rng.choice(["refactor_every", "adaptive"]))
    else:
        n = _log_int(rng, 100, 8000)
        rows = _log_int(rng, 60, min(8000, 3200 * 2000 / n))
        opts = _FAST
    return _sweep(None, n, what, rows, limits=what != "injection" and rng.random() < 0.3,
                  host=rng.random() < 0.25, **opts)


# -------------------------------------------------------------------- data
def _spec(n):
    """(branches, PV buses, loads, load scale) of a grid of ``n`` buses: the named grids' own, else between them."""
    by_n = sorted((s[0], s[1] / s[0], s[2] / s[0], s[3] / s[0], s[5]) for s in GRID_SPECS.values())
    for s in by_n:
        if s[0] == n:
            return tuple(int(round(r * n)) for r in s[1:4]) + (s[4],)
    x, xs = math.log(n), [math.log(s[0]) for s in by_n]
    at = [float(np.interp(x, xs, [s[k] for s in by_n])) for k in range(1, 5)]
    # a random network may be weak somewhere: its loads stay further from the collapse than the named grids'
    return max(n - 1, int(at[0] * n)), max(1, int(at[1] * n)), max(1, int(at[2] * n)), 0.4 * at[3]


@functools.lru_cache(maxsize=8)
def _grid(n):
    """The network itself (one per size); its operating point is the seed's."""
    for name, s in GRID_SPECS.items():
        if s[0] == n:
            return grid_by_name(name, 0)
    branches, pv, loads, scale = _spec(n)
    return make_grid(n, branches, pv, loads, seed=0, load_scale=scale)


@functools.lru_cache(maxsize=8)
def _safe_branches(n):
    return n1_branches(_grid(n))


def _operating_point(grid, rng):
    f = rng.uniform(0.9, 1.05) * rng.lognormal(0.0, 0.05, grid.load_p.size)
    lp = grid.load_p * f
    return dataclasses.replace(grid, load_p=lp, load_q=grid.load_q * f,
                               gen_p=grid.gen_p * (lp.sum() / grid.load_p.sum()))


def _rows(case, grid, rng, n_bus, n_rows, what):
    """(p, q) in MW / MVAr or None, and each row's tripped branches or None, of a case's rows."""
    inj = trips = None
    if what in ("injection", "scenario"):
        inj = injection_scenarios(grid, n_rows, seed=int(rng.integers(1 << 30)))
    if what == "n1":
        ids = rng.permutation(grid.n_branch)
        trips = [[int(b)] for b in (ids if n_rows == 0 else np.resize(ids, n_rows))]
    elif what == "scenario":
        # 0 to 2 branches whose single loss keeps the grid connected; a pair may split it
        safe = _safe_branches(n_bus)
        k, pick = rng.integers(0, 3, n_rows), rng.integers(0, safe.size, (n_rows, 2))
        trips = [sorted({int(safe[b]) for b in pick[r, :k[r]]}) for r in range(n_rows)]
    return inj, trips


def _definition(case, seed):
    """A sweep-like case's grid at its operating point and its rows (one pair per grid), from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "multi":
        out = []
        for n in map(int, case["grids"].split(",")):
            g = _operating_point(_grid(n), rng)
            out.append((g,) + _rows(case, g, rng, n, case["rows"], "scenario"))
        return out
    n = case["n_bus"]
    # a trained network belongs to one base case: its rows differ by the seed, its operating point does not
    g = _grid(n) if case.get("start") == "learned" else _operating_point(_grid(n), rng)
    if kind == "single":
        to = _operating_point(_grid(n), rng)
        return [(g, to.sbus(), None)]
    return [(g,) + _rows(case, g, rng, n, case["rows"], "injection" if kind == "grad" else case["what"])]


@functools.lru_cache(maxsize=2)
def _learned(n):
    """The trained network a program keeps for its grid."""
    ls = LearnedStart(_grid(n), hidden=1024, layers=2, seed=0)
    ls.train(n_rows=8192, epochs=20, batch=1024, seed=7, broad=0.5)
    return ls


def _network(case, seed):
    """bf16 inputs, fp32 targets and fp32 weights of a network case (CPU generator: the same on every machine)."""
    gen = torch.Generator().manual_seed(seed)
    up = lambda v: (v + 127) // 128 * 128  # noqa: E731
    L, h, rows = case["layers"], up(case["hidden"]), up(case["rows"])
    dims = [case["n_in"]] + [h] * L + [case["n_out"]]
    w = [torch.randn(dims[k + 1], dims[k], generator=gen) / math.sqrt(dims[k]) for k in range(L + 1)]
    b = [0.1 * torch.randn(dims[k + 1], generator=gen) for k in range(L + 1)]
    x = torch.zeros(rows, case["n_in"])
    x[:case["rows"]] = torch.randn(case["rows"], case["n_in"], generator=gen)
    t = torch.zeros(rows, case["n_out"])
    t[:case["rows"]] = torch.randn(case["rows"], case["n_out"], generator=gen)
    return x.cuda().to(torch.bfloat16), t.cuda(), [v.cuda() for v in w], [v.cuda() for v in b]


# ----------------------------------------------------------------- prepare
def _facade(grid, inj, trips, opts, limits=False, place=True):
    cls = gs.InjectionSweepGPU if trips is None else (
        gs.ContingencyAnalysisGPU if inj is None else gs.ScenarioSweepGPU)
    f = cls(grid.as_tuple(), init_from_n_powerflow=False, **opts)
    f.set_branch_data(*grid.branch_data())
    if limits:
        f.set_branch_limits(np.full(grid.n_branch, 60.0), SN)
    if place:
        _place(f, inj, trips)
    return f


def _place(f, inj, trips):
    if inj is not None:
        f.set_injections(inj[0], inj[1], SN)
    if trips is not None:
        (f.add_contingencies_by_branch_id if inj is None else f.set_topology)(trips)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "gradients"):
        x, t, w, b = _network(case, seed)
        net = WarmStartMLP(case["n_in"], case["n_out"], hidden=case["hidden"], layers=case["layers"])
        net.master.zero_()
        for k in range(case["layers"] + 1):
            net.W(k)[:w[k].shape[0], :w[k].shape[1]] = w[k]
            net.b(k)[:b[k].shape[0]] = b[k]
        net.wb.copy_(net.master)
        return dict(case=case, net=net, x=net.device_inputs(x), t=net.device_targets(t))
    parts = _definition(case, seed)
    if kind == "single":
        g, to, _ = parts[0]
        ac = gs.AcPfGPU(g.as_tuple(), precision=case["precision"], init_from_n_powerflow=False)
        return dict(case=case, ac=ac, start=ac.solve(), to=to)
    if kind == "multi":
        return dict(case=case, sweeps=[_facade(g, inj, trips, _FAST) for g, inj, trips in parts])
    g, inj, trips = parts[0]
    if kind == "grad":
        f = _facade(g, inj, trips, dict(precision="fp64", scheduling="continuous", nb_iter=10, tol=1e-10))
        rng = np.random.default_rng(seed + 1)
        dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
        return dict(case=case, sweep=f, p=dev(inj[0]).requires_grad_(True), q=dev(inj[1]).requires_grad_(True),
                    wm=dev(rng.standard_normal((case["rows"], g.n_bus))),
                    wa=dev(rng.standard_normal((case["rows"], g.n_bus))))
    opts = {k: case[k] for k in ("precision", "scheduling", "strategy", "nb_iter")}
    f = _facade(g, inj, trips, opts, case["limits"], place=not case["host"])
    if case["host"]:
        f.results_to_host = True
    if case["start"] == "learned":
        f.set_learned_start(_learned(case["n_bus"]))
    return dict(case=case, sweep=f, inj=inj, trips=trips)


# --------------------------------------------------------------------- run
def _on_device(f):
    # the capsules alias the facade's buffers, which its next compute() writes and its end frees: what is kept is copied
    return dict(v=torch.from_dlpack(f.results_dlpack("v")).clone(),
                status=torch.from_dlpack(f.results_dlpack("status")).clone())


def run(state):
    kind = state["case"]["kind"]
    if kind == "predict":
        return state["net"].predict(state["x"])
    if kind == "gradients":
        grads, loss = state["net"].gradients(state["x"], state["t"])
        return dict(grads=grads, loss=loss)
    if kind == "single":
        state["ac"].resolve(state["start"], state["to"])
        return state["ac"].solve()
    if kind == "multi":
        gs.compute_many(state["sweeps"])
        return [_on_device(f) for f in state["sweeps"]]
    if kind == "grad":
        v = batch_power_flow(state["p"], state["q"], state["sweep"], SN)
        loss = (state["wm"] * v.abs()).sum() + (state["wa"] * torch.angle(v)).sum()
        dp, dq = torch.autograd.grad(loss, (state["p"], state["q"]))
        return dict(v=v, loss=loss, dp=dp, dq=dq)
    f = state["sweep"]
    if state["case"]["host"]:
        _place(f, state["inj"], state["trips"])
        f.compute()
        v, _, status, _ = f.results_view()
        out = dict(v=v, status=status)
    else:
        f.compute()
        out = _on_device(f)
    if state["case"]["limits"]:
        out["loading"], out["over"], out["worst"] = f.branch_loading()
    return out


# --------------------------------------------------------- work, tolerance
def _n_rows(case):
    return case["rows"] or _spec(case["n_bus"])[0]


def work(case):
    kind = case["kind"]
    if kind in ("predict", "gradients"):
        i, o, h, L, r = case["n_in"], case["n_out"], case["hidden"], case["layers"], case["rows"]
        weights = i * h + (L - 1) * h * h + h * o
        if kind == "predict":
            return {"bytes": 2 * weights + 2 * r * i + 4 * r * o, "flops": 2 * r * weights}
        return {"bytes": 2 * weights + 2 * r * i + 4 * r * o + 4 * weights, "flops": 2 * r * (3 * weights - i * h)}
    if kind == "multi":
        parts = [work(dict(_sweep(None, int(n), "scenario", case["rows"], **_FAST))) for n in case["grids"].split(",")]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["n_bus"]
    rows = 1 if kind == "single" else _n_rows(case)
    what = {"single": "injection", "grad": "injection"}.get(kind, case.get("what"))
    nbytes = 16 * n * rows * (1 if what == "n1" else 2)
    if case.get("limits"):
        nbytes += 4 * rows * _spec(n)[0]
    # one factorization: the near-dense last block that any elimination order leaves on these grids (about
    # 0.36 n wide up to 2000 buses, then growing as sqrt(n)); one step without one: the mismatch's complex products
    # over Ybus and two products per factor entry outside of it
    dense = 0.26 * n if n <= 2000 else 520.0 * math.sqrt(n / 2000)
    lu, step = 2.0 / 3.0 * dense ** 3, 8 * (n + 2 * _spec(n)[0]) + 2 * dense ** 2
    if kind == "single":
        flops = 3 * (lu + step)
    elif kind == "grad":
        flops = rows * (4 * (lu + step) + lu + step)
        nbytes *= 2
    elif case["strategy"] == "base_chord":
        flops = rows * 4 * step
    else:
        flops = rows * (1 if case["strategy"] == "adaptive" else min(case["nb_iter"], 4)) * (lu + step)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    # fp32 sums, activations (and their gradients) rounded to bf16: 2e-3 and 3e-3 off the 64-bit result
    if kind == "predict":
        return {"rel": 5e-3, "max": 5e-2}
    if kind == "gradients":
        return {"rel": 1e-2, "max": 1e-1}
    if case.get("limits"):
        return {"rel": 1e-6, "max": 1e-5}  # loadings are fp32
    # a row is done when its mismatch is below 1e-8 pu, which leaves its voltages up to about 1e-7 pu apart
    return {"rel": 1e-8, "max": 1e-6}


# ------------------------------------------------------------------- exact
class _Exact:
    """Newton's method in 64-bit torch for the rows of one grid: one dense Jacobian at the base case, its inverse
    applied to every row until the mismatch is at rounding level, rows it does not bring there solved one by one."""

    def __init__(self, g, v0=None):
        dev = "cuda"
        Y = g.Ybus.tocsr()
        self.g, self.n = g, g.n_bus
        self.col = torch.as_tensor(Y.indices.astype(np.int64), device=dev)
        self.row = torch.as_tensor(np.repeat(np.arange(self.n), np.diff(Y.indptr)), device=dev)
        self.val = torch.as_tensor(Y.data, device=dev)
        crow = torch.as_tensor(Y.indptr.astype(np.int64), device=dev)
        self.G, self.B = (torch.sparse_csr_tensor(crow, self.col, v.contiguous(), (self.n, self.n))
                          for v in (self.val.real, self.val.imag))
        pv, pq = np.asarray(g.pv, np.int64), np.asarray(g.pq, np.int64)
        self.pvpq = torch.as_tensor(np.sort(np.concatenate([pv, pq])), device=dev)
        self.pq = torch.as_tensor(pq, device=dev)
        self.f, self.t = (torch.as_tensor(np.asarray(a, np.int64), device=dev) for a in (g.branch_from, g.branch_to))
        self.y = [torch.as_tensor(a, device=dev) for a in (g.yff, g.yft, g.ytf, g.ytt)]
        self.base_s = torch.as_tensor(g.sbus(), device=dev)[None]
        v = torch.as_tensor(g.vinit(), device=dev)[None]
        for _ in range(12):
            f = self.mismatch(v, self.base_s)
            if f.abs().max() < 1e-12:
                break
            v = self.update(v, torch.linalg.solve(self.jacobian(v[0]), f[0])[None])
        self.base_v = v

    def current(self, v, trips=None):
        vr, vi = v.real.T.contiguous(), v.imag.T.contiguous()
        i = torch.complex(self.G @ vr - self.B @ vi, self.G @ vi + self.B @ vr).T.contiguous()
        if trips is not None:
            r, b = trips
            f, t = self.f[b], self.t[b]
            yff, yft, ytf, ytt = (y[b] for y in self.y)
            i.index_put_((r, f), -(yff * v[r, f] + yft * v[r, t]), accumulate=True)
            i.index_put_((r, t), -(ytf * v[r, f] + ytt * v[r, t]), accumulate=True)
        return i

    def mismatch(self, v, s, trips=None):
        d = v * self.current(v, trips).conj() - s
        return -torch.cat([d.real[:, self.pvpq], d.imag[:, self.pq]], 1)

    def jacobian(self, v, trip=()):
        val = self.val
        if len(trip):
            val = val.clone()
            for b in trip:
                f, t = int(self.f[b]), int(self.t[b])
                for y, i, j in zip(self.y, (f, f, t, t), (f, t, f, t)):
                    val[(self.row == i) & (self.col == j)] -= y[b]
        i_bus = torch.zeros(self.n, dtype=v.dtype, device=v.device).index_add_(0, self.row, val * v[self.col])
        u = v / v.abs()
        dva = -1j * v[self.row] * (val * v[self.col]).conj()
        dvm = v[self.row] * (val * u[self.col]).conj()
        diag = self.row == self.col
        dva = dva + torch.where(diag, 1j * v[self.row] * i_bus.conj()[self.row], 0)
        dvm = dvm + torch.where(diag, i_bus.conj()[self.row] * u[self.row], 0)
        n_a = self.pvpq.numel()
        ia = torch.full((self.n,), -1, device=v.device)
        im = ia.clone()
        ia[self.pvpq] = torch.arange(n_a, device=v.device)
        im[self.pq] = n_a + torch.arange(self.pq.numel(), device=v.device)
        J = torch.zeros(n_a + self.pq.numel(), n_a + self.pq.numel(), dtype=torch.float64, device=v.device)
        for rows, cols, x in ((ia, ia, dva.real), (ia, im, dvm.real), (im, ia, dva.imag), (im, im, dvm.imag)):
            a, b = rows[self.row], cols[self.col]
            ok = (a >= 0) & (b >= 0)
            J.index_put_((a[ok], b[ok]), x[ok], accumulate=True)
        return J

    def update(self, v, dx):
        n_a = self.pvpq.numel()
        va, vm = torch.angle(v), v.abs()
        va[:, self.pvpq] += dx[:, :n_a]
        vm[:, self.pq] += dx[:, n_a:]
        return torch.polar(vm, va)

    def split(self, trips, n_rows):
        """Rows whose tripped branches split the grid (labels spread along the branches left)."""
        bad = torch.zeros(n_rows, dtype=torch.bool, device="cuda")
        rows = [r for r in range(n_rows) if trips is not None and len(trips[r])]
        for at in range(0, len(rows), 512):
            part = rows[at:at + 512]
            live = torch.ones(len(part), self.f.numel(), dtype=torch.bool, device="cuda")
            for k, r in enumerate(part):
                live[k, torch.as_tensor(trips[r], device="cuda")] = False
            seen = torch.zeros(len(part), self.n, dtype=torch.int8, device="cuda")
            seen[:, 0] = 1
            f, t = self.f.expand(len(part), -1), self.t.expand(len(part), -1)
            before = 0
            while int(seen.sum()) != before:
                before = int(seen.sum())
                seen.scatter_reduce_(1, t, seen.gather(1, f) * live, "amax")
                seen.scatter_reduce_(1, f, seen.gather(1, t) * live, "amax")
            bad[torch.as_tensor(part, device="cuda")] = ~seen.bool().all(1)
        return bad

    def solve(self, s, trips, n_rows, most=150):
        """(v, status) of rows with injections ``s`` (or None) and tripped branches; None when too many rows need a
        Jacobian of their own."""
        s = self.base_s.expand(n_rows, -1) if s is None else s
        self.inv = torch.linalg.inv(self.jacobian(self.base_v[0]))
        bad = self.split(trips, n_rows)
        pair = None
        if trips is not None:
            r = [k for k in range(n_rows) for _ in trips[k]]
            b = [x for k in range(n_rows) for x in trips[k]]
            pair = (torch.as_tensor(r, device="cuda"), torch.as_tensor(b, device="cuda"))
        v = self.base_v.expand(n_rows, -1).clone()
        for _ in range(300):
            f = self.mismatch(v, s, pair)
            f[bad] = 0
            if f.abs().max() < 1e-12:
                break
            v = self.update(v, f @ self.inv.T)
        f = self.mismatch(v, s, pair)
        left = (~(f.abs().amax(1) < 1e-11) & ~bad).nonzero().flatten().tolist()
        if len(left) > most:
            return None
        for r in left:
            x = self.base_v.clone()
            one = None
            if trips is not None and len(trips[r]):
                one = (torch.zeros(len(trips[r]), dtype=torch.int64, device="cuda"),
                       torch.as_tensor(trips[r], device="cuda"))
            for _ in range(10):
                f1 = self.mismatch(x, s[r:r + 1], one)
                if f1.abs().max() < 1e-11:
                    break
                x = self.update(x, torch.linalg.solve(self.jacobian(x[0], trips[r] if one else ()), f1[0])[None])
            v[r] = x[0]
        v[bad] = complex("nan+nanj")
        return v, bad.to(torch.int32) * 3

    def loading(self, v, trips, rate):
        """Branch loadings, their number above 1 and the largest, of solved rows."""
        vf, vt = v[:, self.f], v[:, self.t]
        yff, yft, ytf, ytt = self.y
        s = torch.maximum((vf * (yff * vf + yft * vt).conj()).abs(), (vt * (ytf * vf + ytt * vt).conj()).abs())
        ld = s * SN / rate
        for r, ids in enumerate(trips or ()):
            ld[r, ids] = torch.where(ld[r, ids].isnan(), ld[r, ids], 0.0)
        return ld, ld.amax(1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("predict", "gradients"):
        return _exact_network(case, seed)
    parts = _definition(case, seed)
    if kind == "single":
        g, to, _ = parts[0]
        e = _Exact(g)
        e.base_s = torch.as_tensor(to, device="cuda")[None]
        v = e.base_v
        for _ in range(12):
            f = e.mismatch(v, e.base_s)
            if f.abs().max() < 1e-12:
                break
            v = e.update(v, torch.linalg.solve(e.jacobian(v[0]), f[0])[None])
        return v[0].cpu().numpy()
    out = []
    for g, inj, trips in parts:
        if g.n_bus > 8500:
            out.append(dict(v=None, status=None))  # its dense Jacobian takes too long
            continue
        e = _Exact(g)
        n_rows = len(trips) if trips is not None else inj[0].shape[0]
        s = None if inj is None else torch.complex(*(torch.as_tensor(a, device="cuda") for a in inj)) / SN
        got = e.solve(s, trips, n_rows)
        if got is None:
            if kind != "multi":
                return None
            out.append(dict(v=None, status=None))
            continue
        out.append(dict(v=got[0], status=got[1]))
        if kind == "grad":
            return _exact_grad(case, seed, e, s, got[0])
        if case.get("limits"):
            ld, worst = e.loading(got[0], trips, 60.0)
            out[0].update(loading=ld, worst=worst, over=None)
    if kind == "multi":
        return out
    if case["host"]:
        out[0] = {k: (None if x is None else x.cpu().numpy()) for k, x in out[0].items()}
    return out[0]


def _exact_grad(case, seed, e, s, v):
    """The loss and its gradients: J^T x = dL/d(angle, magnitude) by iterating with the base case's inverse."""
    rng = np.random.default_rng(seed + 1)
    wm, wa = (torch.as_tensor(rng.standard_normal((case["rows"], e.n)), device="cuda") for _ in range(2))
    loss = (wm * v.abs()).sum() + (wa * torch.angle(v)).sum()
    b = torch.cat([wa[:, e.pvpq], wm[:, e.pq]], 1)
    n_a = e.pvpq.numel()
    u = v / v.abs()

    def jt(x):
        # J^T x with J = d(P at pvpq, Q at pq) / d(angle, magnitude): S = V conj(Y V), so for a weight w on P and z
        # on Q the sum is Re(conj(c) S) with c = w + j z
        c = torch.zeros_like(v)
        c[:, e.pvpq] += x[:, :n_a]
        c[:, e.pq] += 1j * x[:, n_a:]
        cur = e.current(v)
        cv = c.conj() * v
        re, im = cv.real.T.contiguous(), cv.imag.T.contiguous()
        yh = torch.complex(e.GT @ re + e.BT @ im, e.GT @ im - e.BT @ re).T
        # along dV: Re(conj(c) dV conj(I)) + Re(conj(c) V conj(Y dV)) = Re(conj(c I + Y^H (conj(c) V)) dV)
        g = c * cur + yh
        da = (g.conj() * 1j * v).real
        dm = (g.conj() * u).real
        return torch.cat([da[:, e.pvpq], dm[:, e.pq]], 1)

    Yt = e.g.Ybus.T.tocsr()
    crow, col = (torch.as_tensor(a.astype(np.int64), device="cuda") for a in (Yt.indptr, Yt.indices))
    e.GT, e.BT = (torch.sparse_csr_tensor(crow, col, torch.as_tensor(np.ascontiguousarray(a), device="cuda"),
                                          (e.n, e.n)) for a in (Yt.data.real, Yt.data.imag))
    x = torch.zeros_like(b)
    for _ in range(200):
        r = b - jt(x)
        if r.abs().max() < 1e-12 * b.abs().max():
            break
        x = x + r @ e.inv
    dp, dq = torch.zeros_like(wm), torch.zeros_like(wm)
    dp[:, e.pvpq] = x[:, :n_a] / SN
    dq[:, e.pq] = x[:, n_a:] / SN
    return dict(v=v, loss=loss, dp=dp, dq=dq)


def _exact_network(case, seed):
    x, t, w, b = _network(case, seed)
    up = lambda v: (v + 127) // 128 * 128  # noqa: E731
    L, o = case["layers"], up(case["n_out"])
    w = [v.to(torch.bfloat16).double().requires_grad_(True) for v in w]
    b = [v.double().requires_grad_(True) for v in b]
    a = x.double()
    for k in range(L + 1):
        a = a @ w[k].T + b[k]
        if k < L:
            a = torch.nn.functional.gelu(a, approximate="none")
    if case["kind"] == "predict":
        y = torch.zeros(a.shape[0], o, dtype=torch.float64, device="cuda")
        y[:, :case["n_out"]] = a.detach()
        return y
    d = a - t.double()
    loss = 0.5 * (2.0 / d.numel()) * d.square().sum()
    got = torch.autograd.grad(loss, w + b)
    grads = []
    for k in range(L + 1):
        dw = torch.zeros(o if k == L else up(w[k].shape[0]), up(w[k].shape[1]), dtype=torch.float64, device="cuda")
        dw[:w[k].shape[0], :w[k].shape[1]] = got[k]
        db = torch.zeros(dw.shape[0], dtype=torch.float64, device="cuda")
        db[:b[k].shape[0]] = got[L + 1 + k]
        grads.append((dw, db))
    return dict(grads=grads, loss=float(d.square().sum()))
