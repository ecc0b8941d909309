"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more of
the same ranges, ``prepare`` what a program holds before the call (grid, plan, inputs on the
GPU or in pinned host memory), ``run`` one pass through the public entry points, ``work`` the
bytes and operations a pass cannot do without and ``exact`` the results in 64 bits from plain
numpy / torch.

Kinds:
  pf     one power flow through a solver object that keeps its plan (``compute_pf`` with the
         method set of KLUSolver / KLUSolverSingleSlack), new injections on an unchanged grid
  n1     contingency analysis, one outage per instance, every instance from the base state;
         ``host``: ``Plan.batch_n1_arrays`` into pinned arrays, else ``pf_batch_device`` with
         inputs and results on the device; Newton in FP64 or mixed precision
  dc     the same batch as a DC power flow (``Plan(dc=True)``), on the device
  fdpf   the same batch as a fast decoupled power flow with the base factors, on the device
  ts     time series: the injection rows assembled on the device (``DeviceAssembly.sbus``), then the
         warm-started chains over them (``DeviceSeries``)
  flows  branch flows of a batch's result rows (``flows_device``: amps and MW, removed
         branches cleared, failed rows treated as zero voltages)

A seed draws another operating point of the grid (another consistent base state, so other
injections and start voltages) and other profiles; the network and a case's contingency list stay,
as they do between two runs of a study.  Voltages are returned whole with the error codes; rows of instances that did not
converge are zero, as the batch computers store them.  Iteration counts are returned by the FP64
forms; in the mixed form an instance whose mismatch lands on the tolerance may legitimately stop a step
earlier or later, so its results are the voltages and the error codes.
"""
import ctypes
import functools

import numpy as np
import torch

from lightsim2grid_b200 import _native as nat
from lightsim2grid_b200 import synthetic
from lightsim2grid_b200.assembly import DeviceAssembly
from lightsim2grid_b200.flows import BranchSet, flows_device, outage_lists
from lightsim2grid_b200.solver import SOLVER_CLASSES, Plan, SolverType
from lightsim2grid_b200.timeseries import DeviceSeries

TOL = 1e-8


def listed():
    return [
        # one power flow of the smallest grid: latency of the host path and of one launch
        dict(name="pf14_fp64", kind="pf", n=14, chords=0, precision=0, distributed=False),
        # one power flow of a national grid with distributed slack: one instance on the whole GPU
        dict(name="pf2848_fp64_dist", kind="pf", n=2848, chords=0, precision=0, distributed=True),
        # security analysis of a small grid from host arrays: a batch of less than two per SM
        dict(name="n1_118_fp64_host", kind="n1", n=118, chords=0, precision=0, distributed=False, cases=186,
             host=True),
        # regional grid in FP64 (the drop-in precision), distributed slack, device resident
        dict(name="n1_1354_fp64_dist", kind="n1", n=1354, chords=0, precision=0, distributed=True, cases=1991,
             host=False),
        # every outage of the national grid from and to host memory, mixed precision: the headline batch
        dict(name="n1_2848_mixed_host", kind="n1", n=2848, chords=0, precision=1, distributed=False, cases=3776,
             host=True),
        # the same in FP64, device resident (the default solver type of the batch computers)
        dict(name="n1_2848_fp64", kind="n1", n=2848, chords=0, precision=0, distributed=False, cases=3776,
             host=False),
        # every outage of the largest grid
        dict(name="n1_6515_mixed", kind="n1", n=6515, chords=0, precision=1, distributed=False, cases=8796,
             host=False),
        # a grid with long-range branches: high LU fill, a dense trailing block
        dict(name="n1_2848c300_mixed", kind="n1", n=2848, chords=300, precision=1, distributed=False, cases=3776,
             host=False),
        # one year of hourly snapshots
        dict(name="ts_2848_mixed", kind="ts", n=2848, chords=0, precision=1, distributed=False, steps=8760),
        # DC and fast decoupled screening of outages
        dict(name="dc_2848", kind="dc", n=2848, chords=0, cases=3776),
        dict(name="fdpf_1354_bx", kind="fdpf", n=1354, chords=0, cases=1991, method=1),
        # flows of every branch after every outage
        dict(name="flows_2848", kind="flows", n=2848, chords=0, rows=3776, amps=True, power=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["pf", "n1", "n1", "n1", "dc", "fdpf", "ts", "flows"])
    if kind == "pf":
        return dict(kind=kind, n=_log_int(rng, 14, 6515), chords=0, precision=rng.randint(0, 1),
                    distributed=rng.random() < 0.5)
    if kind == "n1":
        n = _log_int(rng, 14, 4000)
        # long-range branches on one grid in four, up to the share that the high-fill grids have
        chords = rng.randint(0, n // 9) if rng.random() < 0.25 else 0
        return dict(kind=kind, n=n, chords=chords, precision=rng.randint(0, 1), distributed=rng.random() < 0.3,
                    cases=_log_int(rng, 4, _branches(n)), host=rng.random() < 0.4)
    if kind in ("dc", "fdpf"):
        n = _log_int(rng, 14, 4000 if kind == "dc" else 2000)
        c = dict(kind=kind, n=n, chords=0, cases=_log_int(rng, 4, _branches(n)))
        return dict(c, method=rng.randint(0, 1)) if kind == "fdpf" else c
    if kind == "ts":
        return dict(kind=kind, n=_log_int(rng, 14, 2848), chords=0, precision=rng.randint(0, 1),
                    distributed=rng.random() < 0.3, steps=_log_int(rng, 24, 3000))
    n = _log_int(rng, 14, 4000)
    amps = rng.random() < 0.75
    return dict(kind="flows", n=n, chords=0, rows=_log_int(rng, 1, 4000), amps=amps,
                power=not amps or rng.random() < 0.75)


# ------------------------------------------------------------------ grids
_NAMED = {v[0]: k for k, v in synthetic.GRID_SIZES.items()}


def _branches(n):
    """Branches of a grid of n buses: the named grids' own, else their usual ratio."""
    return synthetic.GRID_SIZES[_NAMED[n]][1] if n in _NAMED else max(n + 1, int(1.34 * n))


@functools.lru_cache(maxsize=8)
def _grid(n, chords):
    """The grid (network data do not depend on the seed of a case) and its true state."""
    if n in _NAMED:
        name = _NAMED[n]
        nb, nbr, npv = synthetic.GRID_SIZES[name]
        return synthetic.make_grid(nb, nbr, npv, seed=synthetic.NAMED_SEEDS[name], chords=chords)
    return synthetic.make_grid(n, _branches(n), max(2, int(0.18 * n)), seed=n, chords=chords)


def _point(grid, V_true, seed):
    """Another operating point: the true state's angles scaled and moved a little, the
    injections consistent with it (the base power flow's solution is known by construction)."""
    rng = np.random.default_rng([seed, grid.n_bus])
    va = np.angle(V_true) * rng.uniform(0.9, 1.0) + 1e-3 * rng.standard_normal(grid.n_bus)
    va -= va[int(grid.get_slack_ids()[0])]
    V = np.abs(V_true) * np.exp(1j * va)
    return V, V * np.conj(grid.get_Ybus() @ V), rng


def _outages(grid, count):
    nb = grid.nb_powerline()
    rng = np.random.default_rng([nb, count])
    return np.arange(nb) if count >= nb else np.sort(rng.choice(nb, size=count, replace=False))


def _coefficients(grid, branches, dc=False):
    one = grid.dc_branch_coeffs if dc else grid.branch_coeffs
    lists = [one([int(b)]) for b in branches]
    ptr = np.zeros(len(lists) + 1, np.int32)
    ptr[1:] = np.cumsum([len(x) for x in lists])
    flat = [c for x in lists for c in x]
    return ptr, nat.as_i32([c[0] for c in flat]), nat.as_i32([c[1] for c in flat]), nat.as_c128([c[2] for c in flat])


# ------------------------------------------------------------------ states
def _device():
    return torch.device("cuda:0")


def _to(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_device())


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed):
    return {"pf": _prepare_pf, "n1": _prepare_n1, "dc": _prepare_n1, "fdpf": _prepare_n1, "ts": _prepare_ts,
            "flows": _prepare_flows}[case["kind"]](case, seed)


def _prepare_pf(case, seed):
    grid, V_true = _grid(case["n"], case["chords"])
    V, S, rng = _point(grid, V_true, seed)
    st = {(0, False): SolverType.GPUNRSingleSlack, (0, True): SolverType.GPUNR,
          (1, False): SolverType.GPUNRMixedSingleSlack, (1, True): SolverType.GPUNRMixed}
    solver = SOLVER_CLASSES[st[case["precision"], case["distributed"]]]()
    fixed = dict(slack_ids=grid.get_slack_ids(), slack_weights=grid.get_slack_weights(), pv=grid.get_pv(),
                 pq=grid.get_pq())
    Y = grid.get_Ybus()
    solver.compute_pf(Y, V, S, max_iter=10, tol=TOL, **fixed)  # the base case: analyses the grid, keeps the plan
    S_new = S * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, grid.n_bus))
    return dict(kind="pf", solver=solver, Y=Y, V0=V, S=S_new, fixed=fixed)


def _prepare_n1(case, seed):
    grid, V_true = _grid(case["n"], case["chords"])
    V, S, _ = _point(grid, V_true, seed)
    kind = case["kind"]
    Y = grid.get_dcYbus() if kind == "dc" else grid.get_Ybus()
    fdpf = grid.get_Bp_Bpp(case["method"]) if kind == "fdpf" else None
    plan = Plan(Y, V, S, grid.get_slack_ids(), grid.get_slack_weights(), grid.get_pv(), grid.get_pq(),
                distributed=case.get("distributed", False), precision=case.get("precision", 0), dc=kind == "dc",
                fdpf=fdpf)
    ptr, rows, cols, vals = _coefficients(grid, _outages(grid, case["cases"]), kind == "dc")
    ncases, max_iter = ptr.size - 1, 40 if kind == "fdpf" else 10
    iters_out = kind != "n1" or case["precision"] == 0
    if case.get("host"):
        out = (_pinned(ncases * grid.n_bus * 2, torch.float64).view(np.complex128).reshape(ncases, grid.n_bus),
               *(_pinned(ncases, torch.int32) for _ in range(3)))
        return dict(kind="n1_host", plan=plan, args=(ptr, rows, cols, vals, V, S, max_iter, TOL), out=out,
                    iters_out=iters_out)
    lib = nat.load()
    cap = max(int(ptr[-1]), 1)
    solvable, optr = np.zeros(ncases, np.int32), np.zeros(ncases + 1, np.int32)
    opos, oval = np.zeros(cap, np.int32), np.zeros(cap, np.complex128)
    nw = lib.pf_n1_prepare(plan.handle, ncases, nat.ptr(ptr, nat.i32p), nat.ptr(rows, nat.i32p),
                           nat.ptr(cols, nat.i32p), nat.cptr(vals), nat.ptr(solvable, nat.i32p),
                           nat.ptr(optr, nat.i32p), nat.ptr(opos, nat.i32p), nat.cptr(oval), cap)
    if nw < 0:
        raise RuntimeError(nat.last_error(lib))
    ninst = int(solvable.sum())
    order = np.zeros(max(ninst, 1), np.int32)
    nat.check(lib.pf_n1_order(plan.handle, ninst, nat.ptr(optr, nat.i32p), nat.ptr(opos, nat.i32p), nat.cptr(oval),
                              nat.cptr(V), nat.ptr(order, nat.i32p)), "pf_n1_order", lib)
    dev = _device()
    d = dict(V0=_to(V.view(np.float64)), S=_to(S.view(np.float64)), optr=_to(optr[:ninst + 1]),
             opos=_to(opos[:max(nw, 1)]), oval=_to(oval[:max(nw, 1)].view(np.float64)), jf=_to(order[:max(ninst, 1)]),
             jc=torch.ones(max(ninst, 1), dtype=torch.int32, device=dev),
             V=torch.zeros((max(ninst, 1), grid.n_bus), dtype=torch.complex128, device=dev),
             it=torch.zeros(max(ninst, 1), dtype=torch.int32, device=dev),
             er=torch.zeros(max(ninst, 1), dtype=torch.int32, device=dev))
    batch = nat.PfDeviceBatch(n_inst=ninst, V0=d["V0"].data_ptr(), v0_stride=0, Sbus=d["S"].data_ptr(), sbus_stride=0,
                              ovr_ptr=d["optr"].data_ptr(), ovr_pos=d["opos"].data_ptr(), ovr_val=d["oval"].data_ptr(),
                              max_iter=max_iter, tol=TOL, chain=0, job_first=d["jf"].data_ptr(),
                              job_count=d["jc"].data_ptr(), njobs=ninst, Vout=d["V"].data_ptr(),
                              iters=d["it"].data_ptr(), errs=d["er"].data_ptr())
    return dict(kind="n1", plan=plan, d=d, batch=batch, iters_out=iters_out,
                zero=torch.zeros((), dtype=torch.complex128, device=dev))


def _prepare_ts(case, seed):
    grid, V_true = _grid(case["n"], case["chords"])
    V, S, _ = _point(grid, V_true, seed)
    plan = Plan(grid.get_Ybus(), V, S, grid.get_slack_ids(), grid.get_slack_weights(), grid.get_pv(), grid.get_pq(),
                distributed=case["distributed"], precision=case["precision"])
    # around 0.8 of the grid's injections: the daily peaks stay below the grids' loadability
    gen_p, _, load_p, load_q = synthetic.time_series_injections(grid, case["steps"], seed=seed + 1, level=0.8)
    series = DeviceSeries(plan, np.zeros((case["steps"], grid.n_bus), np.complex128), V, plan.info()["grid"], _device(),
                          max_iter=10, tol=TOL)
    return dict(kind="ts", asm=DeviceAssembly(plan, grid, _device()), series=series,
                inj=[_to(a) for a in (gen_p, load_p, load_q)], iters_out=case["precision"] == 0)


def _prepare_flows(case, seed):
    grid, V_true = _grid(case["n"], case["chords"])
    dev = _device()
    rows, nb = case["rows"], grid.nb_powerline()
    gen = torch.Generator(device=dev).manual_seed(seed)
    rng = np.random.default_rng([seed, rows])
    mag = 1.0 + 0.01 * torch.randn((rows, grid.n_bus), generator=gen, device=dev, dtype=torch.float64)
    ang = 0.02 * torch.randn((rows, grid.n_bus), generator=gen, device=dev, dtype=torch.float64)
    V = _to(V_true)[None, :] * torch.polar(mag, ang)
    errs = (rng.random(rows) < 0.01).astype(np.int32) * 2  # TooManyIterations
    removed = rng.integers(0, nb, rows)
    ptr, ids = outage_lists([[int(b)] for b in removed])
    branches = BranchSet(grid)
    struct, keep = branches.device(dev)
    out = [torch.empty((rows, nb), dtype=torch.float64, device=dev) if case[k] else None for k in ("amps", "power")]
    return dict(kind="flows", struct=struct, keep=keep, n=grid.n_bus, rows=rows, V=V, errs=_to(errs), ptr=_to(ptr),
                ids=_to(ids), out=out, host=(branches, errs, removed))


# ------------------------------------------------------------------ passes
def run(s):
    kind = s["kind"]
    if kind == "pf":
        ok = s["solver"].compute_pf(s["Y"], s["V0"], s["S"], max_iter=10, tol=TOL, **s["fixed"])
        return dict(V=s["solver"].get_V(), converged=bool(ok))
    if kind == "n1_host":
        V, conv, iters, errs = s["plan"].batch_n1_arrays(*s["args"], out=s["out"])
        res = dict(V=V, converged=conv, errors=errs)
        return dict(res, iterations=iters) if s["iters_out"] else res
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "n1":
        lib = nat.load()
        nat.check(lib.pf_batch_device(s["plan"].handle, ctypes.byref(s["batch"]), stream), "pf_batch_device", lib)
        d = s["d"]
        res = dict(V=torch.where((d["er"] == 0)[:, None], d["V"], s["zero"]), errors=d["er"])
        return dict(res, iterations=d["it"]) if s["iters_out"] else res
    if kind == "ts":
        d = s["series"].d
        s["asm"].sbus(*s["inj"], stream, out=d["S"])
        s["series"].launch(stream)
        res = dict(V=d["V"], errors=d["er"], S=d["S"])
        return dict(res, iterations=d["it"]) if s["iters_out"] else res
    amps, power = s["out"]
    flows_device(s["struct"], s["n"], s["V"].data_ptr(), s["rows"], stream, errs_ptr=s["errs"].data_ptr(),
                 out_ptr=s["ptr"].data_ptr(), out_ids=s["ids"].data_ptr(),
                 amps_ptr=amps.data_ptr() if amps is not None else 0, p_ptr=power.data_ptr() if power is not None else 0)
    return dict(amps=amps, power=power)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    n, kind = case["n"], case["kind"]
    nb = _branches(n)
    nnz = n + 2 * nb                      # Ybus entries
    m = int(1.8 * n)                      # unknowns of the Newton system
    # one Newton step: mismatch (8 operations per Ybus entry), J (16 per entry), refactorisation
    # (about 40 multiply-adds per unknown at the named grids' fill; the chords' dense block on
    # top) and substitutions (20 operations per unknown), voltage update (40 per bus)
    dense = 0.34 * (1.3 * case["chords"]) ** 3
    step = 24 * nnz + 100 * m + 40 * n + dense
    if kind == "flows":
        outs = (1 if case["amps"] else 0) + (1 if case["power"] else 0)
        return dict(bytes=case["rows"] * (16 * n + 8 * nb * outs) + 49 * nb, flops=30 * case["rows"] * nb)
    if kind == "pf":
        return dict(bytes=48 * n + 20 * nnz, flops=3 * step)
    if kind == "ts":
        # injections read, rows of Sbus and V written; about two steps per warm-started snapshot
        return dict(bytes=case["steps"] * (16 * n + 32 * n), flops=case["steps"] * 2 * step)
    count = case["cases"]
    rows = dict(bytes=count * (16 * n + 80) + 32 * n + 20 * nnz)
    if kind == "dc":
        return dict(rows, flops=count * (2 * nnz + 40 * n))
    if kind == "fdpf":
        return dict(rows, flops=count * 20 * (2 * 12 * nnz + 60 * n))
    return dict(rows, flops=count * 3 * step)


# ------------------------------------------------------------------ results in 64 bits
def _newton(Y, V0, S, pv, pq, steps=12):
    """Newton-Raphson on dense float64 tensors, one slack (bus of neither list), run well past
    the engine's tolerance.  Y: (batch, n, n) complex; returns (V, mismatch) per batch entry."""
    pvpq = torch.cat([pv, pq])
    npvpq = pvpq.numel()
    Vm, Va = V0.abs(), V0.angle()
    best, norm = V0, None
    for _ in range(steps):
        V = torch.polar(Vm, Va)
        I = torch.einsum("bij,bj->bi", Y, V)
        F = V * I.conj() - S
        f = torch.cat([F.real[:, pvpq], F.imag[:, pq]], 1)
        now = f.abs().amax(1)
        if norm is None:
            best, norm = V, now
        else:
            better = now < norm
            best, norm = torch.where(better[:, None], V, best), torch.where(better, now, norm)
        YV = Y * V[:, None, :]
        dVa = 1j * (torch.diag_embed(V * I.conj()) - V[:, :, None] * YV.conj())
        dVm = (V[:, :, None] * YV.conj()) / Vm[:, None, :] + torch.diag_embed(I.conj() * V / Vm)
        J = torch.cat([torch.cat([dVa.real[:, pvpq][:, :, pvpq], dVm.real[:, pvpq][:, :, pq]], 2),
                       torch.cat([dVa.imag[:, pq][:, :, pvpq], dVm.imag[:, pq][:, :, pq]], 2)], 1)
        dx = torch.linalg.solve_ex(J, f[:, :, None])[0][:, :, 0]
        Va, Vm = Va.clone(), Vm.clone()
        Va[:, pvpq] -= dx[:, :npvpq]
        Vm[:, pq] -= dx[:, npvpq:]
        del dVa, dVm, J, YV
    return best, norm


def exact(case, seed):
    kind = case["kind"]
    grid, V_true = _grid(case["n"], case["chords"])
    n = grid.n_bus
    if kind == "flows":
        return _exact_flows(case, seed)
    if kind == "ts":
        gen_p, _, load_p, load_q = synthetic.time_series_injections(grid, case["steps"], seed=seed + 1, level=0.8)
        S = np.zeros((case["steps"], n), np.complex128)
        S[:, grid.gen_bus] += gen_p  # one generator, one load per bus
        S[:, grid.load_bus] -= load_p + 1j * load_q
        return dict(V=None, errors=None, S=S.view(np.float64).ravel(), iterations=None)
    dev = _device()
    V, S, rng = _point(grid, V_true, seed)
    pv, pq = _to(grid.get_pv()), _to(grid.get_pq())
    if kind == "pf":
        if n > 3000:
            return None
        S_new = S * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, n))
        Y = _to(grid.get_Ybus().toarray())[None]
        got, norm = _newton(Y, _to(V)[None], _to(S_new)[None], pv, pq, steps=6)
        return dict(V=got[0].cpu().numpy(), converged=None) if float(norm[0]) < 1e-10 else None
    branches = _outages(grid, case["cases"])
    if kind == "dc":
        if n > 3000:
            return None
        return _exact_dc(case, grid, V, S, branches)
    if n > 300 or kind == "fdpf":
        return None  # a dense Newton per outage would take minutes
    Y0 = _to(grid.get_Ybus().toarray())
    rows, conv = [], []
    for lo in range(0, branches.size, 64):
        part = branches[lo:lo + 64]
        Y = Y0.repeat(part.size, 1, 1)
        alive = []
        for i, b in enumerate(part):
            for r, c, y in grid.branch_coeffs([int(b)]):
                Y[i, r, c] -= complex(y)
            alive.append(_connected(grid, int(b)))
        got, norm = _newton(Y, _to(V)[None].repeat(part.size, 1), _to(S)[None].repeat(part.size, 1), pv, pq)
        rows.append(got)
        conv.append((torch.tensor(alive, device=dev), norm < 1e-10))
    got, alive, ok = torch.cat(rows), torch.cat([c[0] for c in conv]), torch.cat([c[1] for c in conv])
    if not bool(ok[alive].all()):
        return None  # an outage without a solution: its zero row is not a computed number
    got = torch.where(alive[:, None], got, torch.zeros((), dtype=got.dtype, device=dev))
    if case["host"]:
        return dict(V=got.cpu().numpy(), converged=None, errors=None, iterations=None)
    return dict(V=got[alive].cpu().numpy() if bool(alive.any()) else None, errors=None, iterations=None)


def _connected(grid, out):
    """Whether every bus is reached without branch `out`."""
    n = grid.n_bus
    nbrs = [[] for _ in range(n)]
    for k, (f, t) in enumerate(zip(grid.line_from, grid.line_to)):
        if k != out:
            nbrs[int(f)].append(int(t))
            nbrs[int(t)].append(int(f))
    seen, todo = {0}, [0]
    while todo:
        for b in nbrs[todo.pop()]:
            if b not in seen:
                seen.add(b)
                todo.append(b)
    return len(seen) == n


def _exact_dc(case, grid, V, S, branches):
    n, slack = grid.n_bus, int(grid.get_slack_ids()[0])
    keep = _to(np.array([b for b in range(n) if b != slack]))
    B = _to(grid.get_dcYbus().toarray().real)[keep][:, keep]
    f, t = grid.line_from[branches], grid.line_to[branches]
    # theta of every outage from the base inverse by the rank-one update of its branch
    A = torch.zeros((n, branches.size), dtype=torch.float64, device=_device())
    col = torch.arange(branches.size, device=_device())
    A[_to(f), col] = 1.0
    A[_to(t), col] = -1.0
    A = A[keep]
    X = torch.linalg.solve(B, torch.cat([_to(S.real)[keep][:, None], A], 1))
    base, W = X[:, :1], X[:, 1:]
    y = _to(1.0 / grid.line_x[branches])
    den = 1.0 - y * (A * W).sum(0)
    solvable = den.abs() > 1e-6
    theta = base + W * (y * (A * base).sum(0) / den)[None, :]
    va = torch.zeros((n, branches.size), dtype=torch.float64, device=_device())
    va[keep] = theta
    va += float(np.angle(V[slack]))
    out = torch.polar(_to(np.abs(V))[:, None].expand(-1, branches.size).contiguous(), va).T[solvable]
    return dict(V=out.contiguous().cpu().numpy(), errors=None, iterations=None)


def _exact_flows(case, seed):
    s = _prepare_flows(case, seed)
    br, errs, removed = s["host"]
    E = s["V"].clone()
    E[_to(errs) != 0] = 0.0
    ef, et = E[:, _to(br.from_.astype(np.int64))], E[:, _to(br.to.astype(np.int64))]
    flow = ef * (_to(br.yff)[None, :] * ef + _to(br.yft)[None, :] * et).conj()
    amps = flow.abs() * br.sn_mva / (np.sqrt(3.0) * ef.abs() * _to(br.vn_kv_from)[None, :])
    power = flow.real * br.sn_mva
    at = (torch.arange(case["rows"], device=_device()), _to(removed))
    amps[at] = torch.where(amps[at].isfinite(), torch.zeros_like(amps[at]), amps[at])
    power[at] = 0.0
    return dict(amps=amps if case["amps"] else None, power=power if case["power"] else None)
