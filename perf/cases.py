"""The work that users of this framework have it do, as cases that can be timed.

Every case is a multigrid Euler solve (or a stream of them) on seeded meshes of
the framework's own workload family: a jittered lattice of nx x ny x nz nodes with
its coarse levels, ids randomly permuted as a mesh file's are, or in lattice order
as after renumbering.  Freestream Mach 0.3-0.85 and angle of attack 0-6 degrees
come from the seed, as do the jitter and the permutations.

  kind     what a program does
  solver   keeps a device-resident Solver: reset, V-cycles, norms, the variables of
           every level fetched into page-locked buffers that it keeps
  solve    mgcfd_solve: a whole solve from and to page-locked host buffers (upload,
           set-up, V-cycles, download)
  batch    keeps a Batch of uneven meshes: reset, V-cycles, every mesh's variables
  loops    drives the reference's V-cycle op_par_loop by op_par_loop (LoopSolver) on
           device dats, the flux calls in FP64 or in the double-word form
  serve    a Server: requests on fresh meshes submitted together, drained, polled
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "mg-cfd-app-op2_gb300"))

import mgcfd  # noqa: E402
from mgcfd import ops  # noqa: E402
from mgcfd.mesh import level_views_from_arrays  # noqa: E402

RK = 3
MAX_NODES = 8_000_000


def listed():
    return [
        # The smallest solves: a few hundred nodes, where launches and latency are everything.
        dict(name="solver_fp64_8", kind="solver", precision="fp64", accumulation="fp64", nx=8, ny=8, nz=8, levels=3,
             cycles=4),
        # The plain FP64 configuration: 48^3 nodes, 3 levels, 10 V-cycles.
        dict(name="solver_fp64_48", kind="solver", precision="fp64", accumulation="fp64", nx=48, ny=48, nz=48,
             levels=3, cycles=10),
        # The headline workload: 200^3 nodes, 4 levels, 25 V-cycles, FP64.
        dict(name="solver_fp64_200", kind="solver", precision="fp64", accumulation="fp64", nx=200, ny=200, nz=200,
             levels=4, cycles=25),
        # The same mesh and cycles in mixed precision (FP32 fluxes, FP64 node sums).
        dict(name="solver_mixed_200", kind="solver", precision="mixed", accumulation="fp64", nx=200, ny=200, nz=200,
             levels=4, cycles=25),
        # Mixed precision with pair sums on a mid-size mesh of odd extents.
        dict(name="solver_pair32_ragged", kind="solver", precision="mixed", accumulation="pair32", nx=61, ny=45,
             nz=83, levels=3, cycles=20),
        # Double-word fluxes (the FP64 bar off the FP64 pipe) on about a million nodes of odd extents.
        dict(name="solver_dw_ragged", kind="solver", precision="dw", accumulation="fp64", nx=131, ny=97, nz=89,
             levels=4, cycles=25),
        # One whole solve from host memory, as a driver that solves each mesh once does.
        dict(name="solve_fp64_64", kind="solve", precision="fp64", accumulation="fp64", nx=64, ny=64, nz=64, levels=3,
             cycles=10),
        # Batched uneven meshes (16 to 96 nodes per axis, 3 levels, 20 V-cycles), both precisions.
        dict(name="batch_fp64", kind="batch", precision="fp64", accumulation="fp64", meshes=12, lo=16, hi=64,
             levels=3, cycles=20),
        dict(name="batch_mixed", kind="batch", precision="mixed", accumulation="fp64", meshes=16, lo=16, hi=96,
             levels=3, cycles=20),
        # The per-loop drop-in at 100^3: the mesh file's scattered numbering in FP64, and a
        # renumbered mesh of odd extents with double-word fluxes.
        dict(name="loops_fp64_100", kind="loops", precision="fp64", nx=100, ny=100, nz=100, numbering="random",
             levels=4, cycles=3),
        dict(name="loops_dw_ragged", kind="loops", precision="dw", nx=115, ny=77, nz=94, numbering="lattice",
             levels=3, cycles=3),
        # Served solves: fresh meshes of 20K nodes and more, mixed precision, small ones in cohorts.
        dict(name="serve_mixed", kind="serve", precision="mixed", accumulation="fp64", requests=12, lo=27, hi=80,
             levels=3, cycles=50),
    ]


def _extents(rng, lo, hi):
    """Three extents whose product is spread over the logarithm of [lo, hi]."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    base = n ** (1.0 / 3.0)
    ext = [max(6, round(base * a)), max(6, round(base * b)), max(6, round(base / (a * b)))]
    while ext[0] * ext[1] * ext[2] > hi:
        ext[ext.index(max(ext))] -= 1
    return ext


def _most_levels(least):
    """Levels a lattice with `least` nodes on its shortest axis can have (at least 2 nodes per axis on each)."""
    levels = 1
    while (least + 1) // 2 >= 2 and levels < 4 and least > 2:
        least = (least + 1) // 2
        levels += 1
    return levels


def draw(rng):
    kind = rng.choice(["solver", "solver", "solver", "solve", "batch", "loops", "serve"])
    if kind == "serve":
        lo = rng.randint(27, 40)
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed", "dw"]), accumulation="fp64",
                    requests=rng.randint(3, 12), lo=lo, hi=rng.randint(lo + 1, 80), levels=rng.choice([3, 4]),
                    cycles=rng.randint(5, 50))
    if kind == "batch":
        lo = rng.randint(6, 24)
        precision = rng.choice(["fp64", "mixed", "mixed", "dw"])
        accumulation = rng.choice(["fp64", "pair32"]) if precision == "mixed" else "fp64"
        return dict(kind=kind, precision=precision, accumulation=accumulation, meshes=rng.randint(2, 24), lo=lo,
                    hi=rng.randint(lo + 1, 96), levels=rng.choice([1, 2, 3]), cycles=rng.randint(2, 20))
    if kind == "loops":
        nx, ny, nz = _extents(rng, 2000, 2_000_000)
        return dict(kind=kind, precision=rng.choice(["fp64", "dw"]), nx=nx, ny=ny, nz=nz,
                    numbering=rng.choice(["random", "lattice"]), levels=rng.randint(1, _most_levels(min(nx, ny, nz))),
                    cycles=rng.randint(1, 5))
    hi = 2_000_000 if kind == "solve" else MAX_NODES
    nx, ny, nz = _extents(rng, 300, hi)
    precision = rng.choice(["fp64", "fp64", "mixed", "dw"])
    accumulation = rng.choice(["fp64", "pair32"]) if precision == "mixed" else "fp64"
    return dict(kind=kind, precision=precision, accumulation=accumulation, nx=nx, ny=ny, nz=nz,
                levels=rng.randint(1, _most_levels(min(nx, ny, nz))), cycles=rng.randint(2, 25))


# Meshes, made on the GPU.

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _lattice(ext, nlevels, g, numbering="random"):
    """Levels of a jittered lattice as dicts of CUDA tensors, in the layout of mgcfd.Level."""
    dev = "cuda"
    h = 1.0 / (max(ext) - 1)
    levels, perms = [], []
    xyz0 = None
    for l in range(nlevels):
        m = list(ext)
        for _ in range(l):
            m = [(e + 1) // 2 for e in m]
        nx, ny, nz = m
        n = nx * ny * nz
        k, j, i = torch.meshgrid(*(torch.arange(e, device=dev) for e in (nz, ny, nx)), indexing="ij")
        idx = [i.reshape(-1), j.reshape(-1), k.reshape(-1)]
        if l == 0:
            xyz0 = torch.stack([v.double() * h for v in idx], 1)
            inner = torch.ones(n, dtype=torch.bool, device=dev)
            for v, e in zip(idx, m):
                inner &= (v > 0) & (v < e - 1)
            xyz0 += (torch.rand(n, 3, dtype=torch.float64, device=dev, generator=g) - 0.5) * (0.4 * h) * inner[:, None]
            xyz = xyz0
        else:
            s = 1 << l
            at = idx[0] * s + ext[0] * (idx[1] * s + ext[1] * (idx[2] * s))
            xyz = xyz0[at]
        p = torch.randperm(n, device=dev, generator=g) if numbering == "random" else torch.arange(n, device=dev)
        perms.append(p)
        hl2 = (h * (1 << l)) ** 2
        q = torch.arange(n, device=dev)
        ends = []
        for v, e, stride in zip(idx, m, (1, nx, nx * ny)):
            a = q[v + 1 < e]
            ends.append(torch.stack([a, a + stride], 1))
        e2n = torch.cat(ends)
        if numbering == "random":
            e2n = e2n[torch.randperm(len(e2n), device=dev, generator=g)]
        else:  # by their first node, as renumbering leaves them
            e2n = e2n[torch.argsort(e2n[:, 0], stable=True)]
        d = xyz[e2n[:, 1]] - xyz[e2n[:, 0]]
        ewt = d / d.norm(dim=1, keepdim=True) * hl2
        bn, bg, bw = [], [], []
        for ax in range(3):
            for side in (0, 1):
                on = q[idx[ax] == (0 if side == 0 else m[ax] - 1)]
                w = torch.zeros(len(on), 3, dtype=torch.float64, device=dev)
                w[:, ax] = -hl2 if side == 0 else hl2
                bn.append(on)
                bg.append(torch.full((len(on),), 0 if ax == 2 and side == 0 else 3, device=dev))
                bw.append(w)
        bn, bg, bw = torch.cat(bn), torch.cat(bg), torch.cat(bw)
        bp = torch.randperm(len(bn), device=dev, generator=g)
        coords = torch.empty_like(xyz)
        coords[p] = xyz
        levels.append(dict(coords=coords, e2n=p[e2n].int(), b2n=p[bn[bp]].int(), grp=bg[bp].int(), ewt=ewt,
                           bwt=bw[bp].contiguous(), n2mg=None, idx=idx, m=m))
    for l in range(nlevels - 1):
        f, c = levels[l], levels[l + 1]
        parent = (f["idx"][0] >> 1) + c["m"][0] * ((f["idx"][1] >> 1) + c["m"][1] * (f["idx"][2] >> 1))
        n2mg = torch.empty(len(parent), dtype=torch.int32, device="cuda")
        n2mg[perms[l]] = perms[l + 1][parent].int()
        f["n2mg"] = n2mg
    for L in levels:
        del L["idx"], L["m"]
    return levels


def _host_levels(levels, pinned=False):
    def host(t):
        if t is None:
            return None
        t = t.contiguous()
        return (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) if pinned else t.cpu()).numpy()

    return [mgcfd.Level(coords=host(L["coords"]), edge_to_nodes=host(L["e2n"]), bnd_to_node=host(L["b2n"]),
                        bnd_group=host(L["grp"]), edge_weights=host(L["ewt"]), bnd_weights=host(L["bwt"]),
                        node_to_mg=host(L["n2mg"])) for L in levels]


def _inputs(case, seed):
    """[(levels, mach, angle of attack)] of a case: one mesh, or the meshes of a batch or of a stream of requests."""
    rng = np.random.default_rng(int(seed))
    g = _generator(int(seed) * 1000003 + 7)
    out = []
    if "nx" in case:
        exts = [(case["nx"], case["ny"], case["nz"])]
    else:
        count = case.get("meshes", case.get("requests"))
        exts = []
        for k in range(count):  # spread over the range's logarithm, each extent a little different
            n = case["lo"] * (case["hi"] / case["lo"]) ** ((k + 0.5) / count)
            exts.append(tuple(max(case["lo"], min(case["hi"], round(n) + d)) for d in (0, k % 2, -(k % 3))))
    for ext in exts:
        levels = _lattice(ext, case["levels"], g, case.get("numbering", "random"))
        out.append((levels, float(rng.uniform(0.3, 0.85)), float(rng.uniform(0.0, 6.0))))
    return out


def _pinned_rows(counts):
    return [torch.empty(n, 5, dtype=torch.float64, pin_memory=True) for n in counts]


def _pointer(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


class _State:
    """What the program holds; `close` gives back what the library keeps for it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        handle = getattr(self, "handle", None)
        if handle is not None:
            handle.close()


def prepare(case, seed):
    kind = case["kind"]
    inputs = _inputs(case, seed)
    levels, mach, aoa = inputs[0]
    opts = {k: case[k] for k in ("precision", "accumulation") if k in case}
    if kind == "solver":
        host = _host_levels(levels)
        return _State(case=case, handle=mgcfd.Solver(host, mach, aoa, **opts),
                      out=_pinned_rows([L.nnodes for L in host]))
    if kind == "solve":
        host = _host_levels(levels, pinned=True)
        out = _pinned_rows([L.nnodes for L in host])
        return _State(case=case, host=host, views=level_views_from_arrays(host), mach=mach, aoa=aoa, out=out,
                      ptrs=(ctypes.POINTER(ctypes.c_double) * len(out))(*[_pointer(t) for t in out]),
                      options=mgcfd.options(**opts), lib=mgcfd._lib.load())
    if kind == "batch":
        host = [_host_levels(levels) for levels, _, _ in inputs]
        handle = mgcfd.Batch(host, [m for _, m, _ in inputs], [a for _, _, a in inputs], **opts)
        return _State(case=case, handle=handle,
                      out=_pinned_rows([sum(L[l].nnodes for L in host) for l in range(case["levels"])]))
    if kind == "loops":
        return _State(case=case, handle=mgcfd.LoopSolver(_host_levels(levels), mach, aoa))
    server = mgcfd.Server(max_active=8, precision=case["precision"], accumulation=case["accumulation"],
                          max_cycles=case["cycles"], batch_max_meshes=8, batch_max_nodes=100_000)
    return _State(case=case, handle=server,
                  requests=[(_host_levels(levels, pinned=True), m, a) for levels, m, a in inputs])


def _fetch_all(handle, out):
    lib = mgcfd._lib.load()
    for l, t in enumerate(out):
        mgcfd._lib.check(lib.mgcfd_solver_fetch(handle._h, l, mgcfd.Q_VARIABLES, _pointer(t)))
    return list(out)


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "solver":
        s = state.handle
        s.reset()
        s.run(case["cycles"])
        status, rms, rho = s.norms()
        return {"status": status, "rms": rms, "rho_rms": rho, "variables": _fetch_all(s, state.out)}
    if kind == "solve":
        mgcfd._lib.check(state.lib.mgcfd_solve(len(state.out), state.views, state.mach, state.aoa, case["cycles"],
                                               ctypes.byref(state.options), state.ptrs))
        return {"variables": list(state.out)}
    if kind == "batch":
        s = state.handle
        s.reset()
        s.run(case["cycles"])
        status = s.synchronize()
        return {"status": status, "variables": _fetch_all(s, state.out)}
    if kind == "loops":
        s = state.handle
        ops.flux_precision(case["precision"])
        s.run(case["cycles"])
        status, rms = s.synchronize()
        ops.flux_precision("fp64")
        return {"status": status, "rms": rms, "variables": [d["var"] for d in s.L],
                "residuals": [d["res"] for d in s.L]}
    server = state.handle
    ids = [server.submit(levels, m, a, want_result=True) for levels, m, a in state.requests]
    server.drain()
    done = {r["id"]: (r, x) for r, x in server.poll()}
    return {"status": [done[i][0]["status"] for i in ids], "cycles": [done[i][0]["cycles"] for i in ids],
            "variables": [done[i][1] for i in ids]}


# What a pass cannot do without.

def _sizes(ext, nlevels):
    """(nodes, edges) per level."""
    out = []
    m = list(ext)
    for _ in range(nlevels):
        n = m[0] * m[1] * m[2]
        out.append((n, sum(n // e * (e - 1) for e in m)))
        m = [(e + 1) // 2 for e in m]
    return out


def work(case):
    """Per smoothing step: three flux sweeps (each edge's weight and ends, each node's state and increments) and
    updates; every transfer reads and writes both levels' states once.  Inputs that a pass uploads and the variables
    that it hands back are counted once."""
    if "nx" in case:
        exts = [(case["nx"], case["ny"], case["nz"])]
    else:
        count = case.get("meshes", case.get("requests"))
        exts = []
        for k in range(count):
            n = case["lo"] * (case["hi"] / case["lo"]) ** ((k + 0.5) / count)
            exts.append(tuple(max(case["lo"], min(case["hi"], round(n) + d)) for d in (0, k % 2, -(k % 3))))
    narrow = case["precision"] == "mixed"
    edge_b, node_b = (24, 32 + 40 + 40) if narrow else (32 + 8, 40 + 40 + 40)
    total_b = total_f = 0.0
    for ext in exts:
        sizes = _sizes(ext, case["levels"])
        last = len(sizes) - 1
        for l, (n, e) in enumerate(sizes):
            steps = 1 if l in (0, last) else 2
            total_b += case["cycles"] * steps * RK * (edge_b * e + node_b * n)
            total_f += case["cycles"] * steps * RK * (54.0 * e + 60.0 * n)
            if l < last:
                total_b += case["cycles"] * 2 * 80 * n
                total_f += case["cycles"] * 20 * n
            total_b += 40 * n
            if case["kind"] in ("solve", "serve"):
                total_b += 24 * n + 32 * e
    return {"bytes": total_b, "flops": total_f}


# The same solve in plain torch, 64 bits throughout.

def _freestream(mach, aoa):
    angle = math.pi / 180.0 * aoa
    rho, pressure = 1.4, 1.0
    speed = mach * math.sqrt(1.4 * pressure / rho)
    u = [speed * math.cos(angle), speed * math.sin(angle), 0.0]
    m = [rho * v for v in u]
    e = rho * (0.5 * speed * speed) + pressure / 0.4
    return [rho] + m + [e]


def _primitives(x):
    rho, m, e = x[:, 0], x[:, 1:4], x[:, 4]
    u = m / rho[:, None]
    p = (1.4 - 1.0) * (e - 0.5 * rho * (u * u).sum(1))
    s = u.norm(dim=1) + torch.sqrt(1.4 * p / rho)
    return u, p, s


def _flux_through(x, u, p, w):
    """w . F of the Euler fluxes of states x."""
    un = (u * w).sum(1)
    f = x * un[:, None]
    f[:, 1:4] += p[:, None] * w
    f[:, 4] += p * un
    return f


def _add_edges(L, x, flux):
    u, p, s = _primitives(x)
    for lo in range(0, len(L["a"]), 1 << 22):  # in pieces, so that the largest mesh fits easily
        a, b, w = (L[k][lo:lo + (1 << 22)] for k in ("a", "b", "w"))
        xa, xb = x[a], x[b]
        f = -0.5 * (_flux_through(xa, u[a], p[a], w) + _flux_through(xb, u[b], p[b], w))
        fac = -w.norm(dim=1) * float(np.float32(0.2)) * 0.5 * (s[a] + s[b])
        f += fac[:, None] * (xa - xb)
        flux.index_add_(0, a, f)
        flux.index_add_(0, b, f, alpha=-1)
    return u, p


def _exact_solve(levels, mach, aoa, cycles):
    """Per level (variables, residuals) after the V-cycles, and the last level-0 norms."""
    ff = torch.tensor(_freestream(mach, aoa), dtype=torch.float64, device="cuda")
    ffu, ffp, _ = _primitives(ff[None])
    L = []
    for lv in levels:
        n = len(lv["coords"])
        a, b = lv["e2n"][:, 0].long(), lv["e2n"][:, 1].long()
        d = lv["coords"][b] - lv["coords"][a]
        dist, area = d.norm(dim=1), lv["ewt"].norm(dim=1)
        vol = torch.zeros(n, dtype=torch.float64, device="cuda")
        vol.index_add_(0, a, dist * area / 6.0)
        vol.index_add_(0, b, dist * area / 6.0)
        bwt = lv["bwt"] * 1e-7
        far = (lv["grp"] >= 3) & (lv["grp"] <= 7)
        wall = lv["grp"] <= 2
        nfar = int(far.sum())
        fffar = _flux_through(ff.expand(nfar, 5).clone(), ffu.expand(nfar, 3), ffp.expand(nfar), bwt[far])
        L.append(dict(n=n, a=a, b=b, w=d / dist[:, None] * area[:, None] / dist[:, None] * 1e-7, vol=vol,
                      wn=lv["b2n"][wall].long(), ww=bwt[wall], fn=lv["b2n"][far].long(), fw=bwt[far], fffar=fffar,
                      x=ff.repeat(n, 1), res=torch.zeros(n, 5, dtype=torch.float64, device="cuda"),
                      up=lv["n2mg"].long() if lv["n2mg"] is not None else None, coords=lv["coords"]))
    norms = (0.0, 0.0)

    def smooth(D):
        old = D["x"]
        sf = (0.5 * D["vol"].pow(1.0 / 3.0) / _primitives(old)[2]).min() / D["vol"]
        x = old
        for rk in range(RK):
            flux = torch.zeros_like(old)
            u, p = _add_edges(D, x, flux)
            wall = torch.zeros(len(D["wn"]), 5, dtype=torch.float64, device="cuda")
            wall[:, 1:4] = D["ww"] * p[D["wn"]][:, None]
            flux.index_add_(0, D["wn"], wall)
            n = D["fn"]
            flux.index_add_(0, n, 0.5 * (D["fffar"] + _flux_through(x[n], u[n], p[n], D["fw"])))
            x = old + (sf / (RK + 1 - rk))[:, None] * flux
        D["x"], D["res"] = x, x - old

    def down_and_up():
        nonlocal norms
        smooth(L[0])
        norms = (float((L[0]["res"].square().sum() / L[0]["n"]).sqrt()),
                 float((L[0]["res"][:, 0].square().sum() / L[0]["n"]).sqrt()))
        for l in range(1, len(L)):
            f, c = L[l - 1], L[l]
            s = torch.zeros(c["n"], 5, dtype=torch.float64, device="cuda").index_add_(0, f["up"], f["x"])
            k = torch.bincount(f["up"], minlength=c["n"])
            c["x"] = torch.where(k[:, None] > 0, s / k.clamp(min=1)[:, None], c["x"])
            smooth(c)
        for l in range(len(L) - 2, -1, -1):
            f, c = L[l], L[l + 1]
            d = (f["coords"] - c["coords"][f["up"]]).abs()
            dm = d.norm(dim=1, keepdim=True)
            f["x"] = f["x"] - torch.cat([dm, d, dm], 1) * (c["res"][f["up"]] - f["res"])
            if l > 0:
                smooth(f)

    for _ in range(cycles):
        down_and_up()
    return [D["x"] for D in L], [D["res"] for D in L], norms


def exact(case, seed):
    kind = case["kind"]
    solved = [_exact_solve(levels, m, a, case["cycles"]) for levels, m, a in _inputs(case, seed)]
    x, res, (rms, rho) = solved[0]
    if kind == "solver":
        return {"status": None, "rms": rms, "rho_rms": rho, "variables": x}
    if kind == "solve":
        return {"variables": x}
    if kind == "batch":
        return {"status": None, "variables": [torch.cat([s[0][l] for s in solved]) for l in range(case["levels"])]}
    if kind == "loops":
        return {"status": None, "rms": rms, "variables": x, "residuals": res}
    return {"status": None, "cycles": None, "variables": [s[0][0] for s in solved]}
