"""The work this framework is used for, as timed cases.

Every case goes through the public Python entry points (``Context``,
``domain.slab_solver``, ``Server``), which call the C ABI one to one.  The
grids run from 32^3, where a solve is launch and synchronisation latency, to
256^3 with 64 right-hand sides, where it is HBM traffic.  Fixed-iteration
runs (``-m K -i`` on the command line, the reference's own example) and runs
to a tolerance are both listed.  BiCGStab runs stop after 16 iterations:
its iterates lose all common digits soon after, whatever computes them.

Kinds:
  solve     one right-hand side in FP64, device vectors (the drop-in call)
  estimate  the probe loop on device probes, many right-hand sides at once
  host      the probe loop from a seed to host arrays (what the CLI does)
  slab      the decomposed solver, all slabs in this process
  server    a handful of jobs through the serving loop
"""
import numpy as np
import torch

import sedi_b200 as S
from sedi_b200 import domain

A = 6.0  # the estimator's stencil: 6 on the diagonal, -1 to each neighbour
FLOPS = {"cg": 21, "pcg": 30, "bicgstab": 38}  # per point and iteration: stencils, updates, dot products


def listed():
    return [
        # The reference's smallest published configuration: 32^3, 50 iterations.
        dict(name="solve_cg_32", kind="solve", solver="cg", n1=32, n2=32, n3=32, maxiter=50, tol=1e-9),
        # Odd, unequal edges of a domain that was not chosen for the hardware.
        dict(name="solve_pcg_odd", kind="solve", solver="pcg", n1=63, n2=47, n3=85, maxiter=50, tol=1e-9),
        dict(name="solve_bicgstab_odd", kind="solve", solver="bicgstab", n1=97, n2=65, n3=51, maxiter=16, tol=1e-9),
        # The drop-in solve at 128^3 to convergence.
        dict(name="solve_cg_128_tol", kind="solve", solver="cg", n1=128, n2=128, n3=128, maxiter=2000, tol=1e-9),
        # One vector larger than L2.
        dict(name="solve_cg_256", kind="solve", solver="cg", n1=256, n2=256, n3=256, maxiter=50, tol=1e-9),
        # The 128^3, 64-probe configuration in mixed precision, to convergence.
        dict(name="est_cg_mixed_128x64_tol", kind="estimate", solver="cg", precision="mixed", n1=128, n2=128, n3=128,
             lanes=64, maxiter=2000, tol=1e-9),
        # The large mixed-precision estimate, bound by HBM.
        dict(name="est_cg_mixed_256x64", kind="estimate", solver="cg", precision="mixed", n1=256, n2=256, n3=256,
             lanes=64, maxiter=50, tol=1e-9),
        # Many probes in FP64: pipelined CG on a mid-size grid, BiCGStab on a ragged one.
        dict(name="est_pcg_fp64_96x32", kind="estimate", solver="pcg", precision="fp64", n1=96, n2=96, n3=96, lanes=32,
             maxiter=50, tol=1e-9),
        dict(name="est_bicgstab_mixed_ragged", kind="estimate", solver="bicgstab", precision="mixed", n1=110, n2=90,
             n3=75, lanes=40, maxiter=16, tol=1e-9),
        # A whole small estimate from a seed: probe generation, solves, host results.
        dict(name="host_cg_fp64_48x16_tol", kind="host", solver="cg", precision="fp64", n1=48, n2=48, n3=48, lanes=16,
             maxiter=2000, tol=1e-9),
        # Two slabs of a decomposed grid.
        dict(name="slab_cg_2", kind="slab", solver="cg", n1=192, n2=160, n3=128, parts=2, maxiter=20, tol=1e-9),
        # Six jobs of mixed sizes through the server.
        dict(name="server_6_jobs", kind="server", jobs=6, edge_lo=32, edge_hi=64, lanes=12, maxiter=2000, tol=1e-8),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "estimate", "estimate", "estimate", "host", "slab", "server"])
    if kind == "server":
        lo = rng.randint(24, 40)
        return dict(kind=kind, jobs=rng.randint(2, 6), edge_lo=lo, edge_hi=rng.randint(lo + 4, 64),
                    lanes=rng.randint(4, 12), maxiter=2000, tol=10.0 ** rng.uniform(-9, -6))
    solver = rng.choice(["cg", "cg", "pcg", "bicgstab"])
    hi = {"solve": 256, "estimate": 160, "host": 80, "slab": 192}[kind]
    c = dict(kind=kind, solver=solver, n1=_log_int(rng, 24, hi), n2=_log_int(rng, 24, hi), n3=_log_int(rng, 24, hi))
    points = c["n1"] * c["n2"] * c["n3"]
    if kind in ("estimate", "host"):
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["lanes"] = max(2, min(_log_int(rng, 4, 64), (1 << (27 if c["precision"] == "mixed" else 26)) // points))
    if kind == "slab":
        c["parts"] = rng.randint(1, 4)
    c["maxiter"] = rng.randint(8, 16) if solver == "bicgstab" else rng.randint(20, 60)
    c["tol"] = 1e-9
    if kind != "slab" and solver == "cg" and rng.random() < 0.4:  # to a tolerance instead
        c["maxiter"], c["tol"] = 2000, 10.0 ** rng.uniform(-9, -6)
    return c


def _dims(case):
    return case["n1"], case["n2"], case["n3"]


def _probes(seed, count, n):
    """+-1 vectors, the right-hand sides the estimator solves for."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.empty((count, n), dtype=torch.float64, device="cuda")
    for k in range(count):
        v[k] = torch.randint(0, 2, (n,), generator=g, device="cuda", dtype=torch.int8).to(torch.float64) * 2.0 - 1.0
    return v


def _jobs(case, seed):
    """The server's job list: (solver, edge, samples, seed, precision)."""
    r = np.random.default_rng(seed)
    out = []
    for k in range(case["jobs"]):
        f = k / max(1, case["jobs"] - 1)
        edge = int(round(case["edge_lo"] + f * (case["edge_hi"] - case["edge_lo"])))
        out.append(("cg" if k % 3 else "pcg", edge, case["lanes"] - k % 3, int(r.integers(1, 2 ** 31)),
                    S.MIXED if k % 2 else S.FP64))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "server":
        return dict(case=case, jobs=_jobs(case, seed), server=S.Server())
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    st = dict(case=case)
    if kind == "slab":
        s = st["solver"] = domain.slab_solver(case["solver"], dims, case["parts"], loopback=True)
        v = _probes(seed, 1, n).view(dims[2], dims[1], dims[0])
        st["x"], st["b"], st["work"] = s.zeros(), s.zeros(), s.work()
        for buf, (first, count) in zip(st["b"], s.ranges):
            buf[1:-1].copy_(v[first:first + count])
        return st
    mixed = case.get("precision") == "mixed"
    st["ctx"] = S.Context(case["solver"], dims, precision=S.MIXED if mixed else S.FP64, batch=case.get("lanes", 1))
    if kind == "solve":
        st["b"] = _probes(seed, 1, n)[0]
        st["x"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        st["stream"] = torch.cuda.Stream()
        st["ctx"].set_stream(st["stream"])  # x = 0 and the solve in one order
    elif kind == "estimate":
        st["probes"] = _probes(seed, case["lanes"], n)
        for k in "Dtq":
            st[k] = torch.empty(n, dtype=torch.float64, device="cuda")
    else:
        st["seed"] = int(seed)
    torch.cuda.synchronize()  # the context's stream does not wait for torch's
    return st


def run(st):
    case = st["case"]
    kind, m, tol = case["kind"], case.get("maxiter"), case.get("tol")
    if kind == "solve":
        with torch.cuda.stream(st["stream"]):
            st["x"].zero_()
            rc, err, it = st["ctx"].solve(st["x"], st["b"], None, m, tol)
        return dict(x=st["x"], rc=rc, iters=it)
    if kind == "estimate":
        r = st["ctx"].estimate_dev(case["lanes"], st["probes"], st["D"], st["t"], st["q"], m, tol)
        return dict(D=st["D"], t=st["t"], q=st["q"], iters=r["iters"], results=r["results"])
    if kind == "host":
        r = st["ctx"].estimate(case["lanes"], st["seed"], m, tol)
        return dict(D=r["D"], t=r["t"], q=r["q"], iters=r["iters"], results=r["results"])
    if kind == "slab":
        for x in st["x"]:
            x.zero_()
        rc, err, it = st["solver"].solve(st["x"], st["b"], m, tol, st["work"])
        return dict(x=[x[1:-1] for x in st["x"]], rc=rc, iters=it)
    srv = st["server"]
    ids = [srv.submit(sol, (e, e, e), k, seed, m, tol, prec) for sol, e, k, seed, prec in st["jobs"]]
    srv.wait()
    return [{k: r[k] for k in ("D", "iters", "results")} for r in (srv.take(i) for i in ids)]


def _iterations(case, edge):
    """Iterations of a run: the fixed count, or what CG takes to reach tol on such a grid."""
    to_tol = 0.42 * edge * -np.log10(case["tol"])
    return int(min(case["maxiter"], to_tol))


def work(case):
    if case["kind"] == "server":
        nbytes = flops = 0.0
        for solver, e, k, _, _ in _jobs(case, 0):
            nbytes += 8.0 * e ** 3
            flops += FLOPS[solver] * float(e) ** 3 * k * _iterations(case, e)
        return {"bytes": nbytes, "flops": flops}
    n = float(case["n1"]) * case["n2"] * case["n3"]
    lanes = case.get("lanes", 1)
    flops = FLOPS[case["solver"]] * n * lanes * _iterations(case, max(_dims(case)))
    # Right-hand sides in (made from the seed on the host path), x or D, t, q out.
    words = {"solve": 2 * n, "slab": 2 * n, "estimate": (lanes + 3) * n, "host": 3 * n}[case["kind"]]
    return {"bytes": 8.0 * words, "flops": flops}


# ---------------------------------------------------------------------------
# The same results from plain torch in 64 bits.
# ---------------------------------------------------------------------------
def _apply(x):
    y = A * x
    y[:, 1:] -= x[:, :-1]
    y[:, :-1] -= x[:, 1:]
    y[:, :, 1:] -= x[:, :, :-1]
    y[:, :, :-1] -= x[:, :, 1:]
    y[:, :, :, 1:] -= x[:, :, :, :-1]
    y[:, :, :, :-1] -= x[:, :, :, 1:]
    return y


def _dot(a, b):
    return (a * b).flatten(1).sum(1)[:, None, None, None]


def _krylov(solver, dims, b, maxiter, tol):
    """x of each right-hand side b[k] from x = 0; a converged one is left as it is."""
    b = b.view(-1, dims[2], dims[1], dims[0])
    x, r, im = torch.zeros_like(b), b.clone(), 1.0 / A
    bb = _dot(b, b)
    live = torch.ones_like(bb)
    if solver == "bicgstab":
        rh, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
        rho = al = om = torch.ones_like(bb)
        for _ in range(maxiter):
            new = _dot(r, rh)
            be = (new / rho) * (al / om)
            rho = new
            p = r + be * (p - om * v)
            v = _apply(p * im)
            al = rho / _dot(v, rh)
            s = r - al * v
            t = _apply(s * im)
            om = _dot(t, s) / _dot(t, t)
            x = x + live * (al * im * p + om * im * s)
            r = s - om * t
            live = live * ((_dot(r, r) / bb).sqrt() > tol)
            if not bool(live.any()):
                break
        return x
    p = r * im
    ru = _dot(r, p)
    for it in range(maxiter):
        s = _apply(p)
        al = live * (ru / _dot(s, p))
        # pipelined CG tests the residual its iteration began with
        rr = _dot(r, r) if solver == "pcg" else None
        x += al * p
        r -= al * s
        u = r * im
        new = _dot(r, u)
        p = u + (new / ru) * p
        ru = new
        live = live * (((_dot(r, r) if rr is None else rr) / bb).sqrt() > tol)
        if it % 8 == 7 and not bool(live.any()):
            break
    return x


def _solutions(solver, dims, b, maxiter, tol):
    n = dims[0] * dims[1] * dims[2]
    step = max(1, (1 << 24) // n)  # right-hand sides at a time
    for k in range(0, b.shape[0], step):
        yield b[k:k + step], _krylov(solver, dims, b[k:k + step], maxiter, tol).view(-1, n)


def _estimate(solver, dims, b, maxiter, tol):
    t, q = 0.0, 0.0
    for v, x in _solutions(solver, dims, b, maxiter, tol):
        t, q = t + (x * v).sum(0), q + (v * v).sum(0)
    return dict(D=t / q, t=t, q=q)


def _seeded(seed, count, n):
    """The estimator's own probes: +-1 from std::mt19937(seed + k), two draws a point."""
    v = np.empty((count, n))
    for k in range(count):
        bits = np.random.Generator(_mt(seed + k)).integers(0, 1 << 32, 2 * n, np.uint32, endpoint=False)
        v[k] = np.where(bits[0::2].astype(np.float64) + bits[1::2].astype(np.float64) * 2.0 ** 32 > 2.0 ** 63, 1.0, -1.0)
    return torch.from_numpy(v).cuda()


def _mt(seed):
    g = np.random.MT19937()
    g._legacy_seeding(int(seed) & 0xFFFFFFFF)  # init_genrand, as std::mt19937 seeds
    return g


def exact(case, seed):
    kind = case["kind"]
    if kind == "server":
        out = []
        for solver, e, k, s, _ in _jobs(case, seed):
            D = _estimate(solver, (e, e, e), _seeded(s, k, e ** 3), case["maxiter"], case["tol"])["D"]
            out.append(dict(D=D, iters=None, results=None))
        return out
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    if kind in ("solve", "slab"):
        x = _krylov(case["solver"], dims, _probes(seed, 1, n), case["maxiter"], case["tol"]).view(n)
        if kind == "solve":
            return dict(x=x, rc=None, iters=None)
        x = x.view(dims[2], dims[1], dims[0])
        cuts = [domain.slab_range(dims[2], case["parts"], s) for s in range(case["parts"])]
        return dict(x=[x[f:f + c] for f, c in cuts], rc=None, iters=None)
    b = _probes(seed, case["lanes"], n) if kind == "estimate" else _seeded(seed, case["lanes"], n)
    return dict(_estimate(case["solver"], dims, b, case["maxiter"], case["tol"]), iters=None, results=None)
