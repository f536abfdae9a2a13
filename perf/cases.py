"""The work that is timed when this package is made faster, and a plain FP64
torch statement of the same work to compare results with.

Each case is one of the ways a program uses the package: a C-level Riemann
call on device rows, steps of one 2D or 3D grid, steps of a parameter sweep
(many uneven grids in one Batch), host-state stepping of a sweep, and a
differentiable rollout with its gradient.  A pass starts from a given state,
takes the steps and reads the state back to the caller's device (or host)
arrays, as a short simulation run does.
"""
import math
import random

import torch

from bonzo_b200 import _lib
from bonzo_b200.adjoint import rollout

RHO, VX, VY, VZ, PR, PSC, BX, BY, BZ = range(9)
GAM = 5.0 / 3.0
SWEEP = (64, 96, 128, 192, 256, 384, 512)  # grid sides of the blast sweep
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _grid(kind, nx, ny, nz, flow, bc, steps, **more):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, flow=flow, bcx=bc[0], bcy=bc[1], bcz=bc[2], steps=steps,
             rsolver="hlld", limiter="vl", charact=0, grav=0.0, graph=True)
    c.update(more)
    return c


def listed():
    return [
        # one row of interface states through the solver: the smallest call
        dict(name="riemann_rows", kind="riemann", n=4096, rsolver="hlld", nvar=9),
        # a quick look at one small blast: launches and host work count
        dict(_grid("grid", 64, 64, 1, "blast", (1, 1, 1), 10), name="blast2d_64"),
        # an odd-sized stratified box with mixed walls, stepped by the host loop
        dict(_grid("grid", 201, 150, 1, "turb", (0, 2, 0), 10, limiter="mc", grav=-0.5, graph=False),
             name="walls2d_201x150"),
        # a production 2D grid with characteristic reconstruction
        dict(_grid("grid", 384, 384, 1, "turb", (0, 0, 0), 8, charact=1), name="charact2d_384"),
        # the uneven blast sweep of the benchmark: 64 grids in one batch
        dict(_grid("sweep", 0, 0, 1, "blast", (1, 1, 1), 10, ninst=64, sizes=2), name="sweep2d_64"),
        # a small ragged sweep with the robust solver
        dict(_grid("sweep", 0, 0, 1, "blast", (1, 2, 1), 20, ninst=24, sizes=-7, rsolver="hll", limiter="mm"),
             name="sweep2d_ragged"),
        # decaying 3D turbulence at the benchmark's size
        dict(_grid("grid", 256, 256, 256, "turb", (0, 0, 0), 4, mach=1.0), name="turb3d_256"),
        # a small odd 3D box with open ends
        dict(_grid("grid", 97, 65, 50, "blast", (1, 0, 2), 6, limiter="mc"), name="blast3d_97x65x50"),
        # 3D conduction (field-aligned heat flux, RKL2 stages every step)
        dict(_grid("grid", 192, 192, 192, "heat", (0, 0, 0), 2, kappa0=0.01, graph=False), name="conduction3d_192"),
        # the hydro build
        dict(_grid("grid", 128, 128, 128, "blast", (1, 1, 1), 6, rsolver="hllc", hydro=True), name="hydro3d_128"),
        # the gradient of a density misfit through 100 steps of a 256^2 vortex
        dict(_grid("rollout", 256, 256, 1, "turb", (0, 0, 0), 100, dt=1e-4, every=10), name="rollout2d_256"),
        # a sweep whose state lives on the host: in, one step, out
        dict(_grid("host", 0, 0, 1, "blast", (1, 1, 1), 1, ninst=16, sizes=3), name="host_sweep2d_16"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("riemann", "grid2", "grid2", "sweep", "sweep", "grid3", "grid3", "heat", "hydro", "rollout",
                       "host"))
    bc = tuple(rng.choice((0, 1, 2)) for _ in range(3))
    lim = rng.choice(("vl", "vl", "mc", "mm"))
    rs = rng.choice(("hlld", "hlld", "hlld", "hll"))
    if kind == "riemann":
        rs, nvar = rng.choice((("hlld", 9), ("hll", 9), ("hllt", 9), ("hllc", 6), ("hll", 6)))
        return dict(kind="riemann", n=_log(rng, 512, 2000000), rsolver=rs, nvar=nvar)
    if kind == "grid2":
        cp = rng.choice((0, 0, 1))
        return _grid("grid", _log(rng, 32, 640), _log(rng, 32, 640), 1, rng.choice(("blast", "turb")), bc,
                     rng.randint(4, 12), rsolver=rs, limiter=lim, charact=cp, grav=rng.choice((0.0, -0.5)),
                     graph=rng.random() < 0.5)
    if kind == "sweep":
        return _grid("sweep", 0, 0, 1, rng.choice(("blast", "turb")), bc, rng.randint(6, 20),
                     ninst=_log(rng, 4, 48), sizes=rng.choice((1, -1)) * rng.randint(1, 99), rsolver=rs, limiter=lim)
    if kind == "grid3":
        return _grid("grid", _log(rng, 24, 200), _log(rng, 24, 200), _log(rng, 24, 200),
                     rng.choice(("blast", "turb")), bc, rng.randint(2, 6), rsolver=rs, limiter=lim,
                     graph=rng.random() < 0.5)
    if kind == "heat":
        return _grid("grid", _log(rng, 24, 180), _log(rng, 24, 180), _log(rng, 24, 180), "heat", (0, 0, 0),
                     rng.randint(1, 3), limiter=lim, kappa0=rng.choice((0.01, 0.003)), graph=False)
    if kind == "hydro":
        return _grid("grid", _log(rng, 24, 160), _log(rng, 24, 160), rng.choice((1, _log(rng, 24, 160))), "blast", bc,
                     rng.randint(2, 8), limiter=lim, rsolver=rng.choice(("hllc", "hll")), hydro=True)
    if kind == "rollout":
        return _grid("rollout", _log(rng, 32, 256), _log(rng, 32, 256), 1, "turb", bc, rng.randint(6, 60), dt=1e-4,
                     every=rng.randint(3, 12), rsolver=rng.choice(("hlld", "hlld", "hll")))
    return _grid("host", 0, 0, 1, "blast", bc, 1, ninst=_log(rng, 4, 16), sizes=rng.choice((1, -1)) * rng.randint(1, 99),
                 rsolver=rs, limiter=lim)


def _dims(case):
    return 3 if case["nz"] > 1 else 2


def _sides(case):
    """(nx, ny, nz) of each grid: a sweep draws squares of the benchmark's
    sides (sizes > 0) or ragged rectangles (sizes < 0)."""
    if case["kind"] not in ("sweep", "host"):
        return [(case["nx"], case["ny"], case["nz"])]
    r = random.Random(abs(case["sizes"]))
    if case["sizes"] > 0:
        return [(s, s, 1) for s in (r.choice(SWEEP) for _ in range(case["ninst"]))]
    return [(_log(r, 40, 200), _log(r, 40, 200), 1) for _ in range(case["ninst"])]


def _bc(case):
    return tuple((case[k], case[k]) for k in ("bcx", "bcy", "bcz"))


def _method(case):
    m = dict(gam=GAM, cour=0.3 if _dims(case) == 3 else 0.4, rsolver=case["rsolver"], limiter=case["limiter"],
             charact_proj=case["charact"])
    if case["grav"]:
        m["grav"] = (0.0, case["grav"], 0.0)
    if case.get("kappa0"):
        m["kappa0"] = case["kappa0"]
    if case.get("hydro"):
        m["hydro"] = True
    return m


def _split(case):
    # the facade's rule: fused tile kernels on 2D PLM grids, the split path elsewhere
    return _dims(case) == 3 or bool(case.get("hydro"))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(*key):
    g = torch.Generator(device="cpu")
    g.manual_seed(hash(tuple(int(k) for k in key)) & 0x7FFFFFFF)
    return g


class _Waves:
    """A smooth random field: a few Fourier modes with kmin <= |k| <= kmax and a
    falling spectrum, of unit rms, evaluated wherever it is asked for."""

    def __init__(self, gen, dims, kmin, kmax, n=12):
        self.k, self.a, self.ph = [], [], []
        while len(self.k) < n:
            k = [int(v) for v in torch.randint(-kmax, kmax + 1, (3,), generator=gen)]
            k = [k[d] if d < dims else 0 for d in range(3)]
            m = math.sqrt(sum(v * v for v in k))
            if kmin <= m <= kmax:
                self.k.append(k)
                self.a.append(m ** -1.8)
                self.ph.append(2 * math.pi * float(torch.rand((), generator=gen)))
        s = math.sqrt(2.0 / sum(a * a for a in self.a))
        self.a = [a * s for a in self.a]

    def at(self, x, y, z, amps=None):
        out = 0.0
        for q, (k, a, ph) in enumerate(zip(self.k, self.a, self.ph)):
            if amps is not None:
                a = a * amps[q]
            arg = (2 * math.pi) * (k[0] * x[None, None, :] + k[1] * y[None, :, None] + k[2] * z[:, None, None]) + ph
            out = out + a * torch.cos(arg)
        return out


def _centres(n, dev):
    return (torch.arange(n, dtype=F64, device=dev) + 0.5) / n


def _faces(n, dev):
    return torch.arange(n + 1, dtype=F64, device=dev) / n


def _initial(case, n, seed, inst, dev="cuda"):
    """Active-cell prim (9, nz, ny, nx) and the three face fields (one more
    face along their own axis): a blast in a weakly stirred medium, turbulence
    (Mach 0.5, or as the case says) in a guide field, or a random temperature field."""
    nx, ny, nz = n
    dims = 3 if nz > 1 else 2
    g = _gen(seed, inst, 77)
    u = lambda a, b: a + (b - a) * float(torch.rand((), generator=g))
    kmax = max(3, min(12, min(nx, ny, nz if dims == 3 else nx) // 8))
    xc, yc, zc = _centres(nx, dev), _centres(ny, dev), _centres(nz, dev)
    xf, yf, zf = _faces(nx, dev), _faces(ny, dev), _faces(nz, dev)
    flow = case["flow"]
    prim = torch.zeros((9, nz, ny, nx), dtype=F64, device=dev)
    scal = lambda: _Waves(g, dims, 1, kmax, 6).at(xc, yc, zc)
    vamp = {"blast": 0.05, "turb": case.get("mach", 0.5), "heat": 0.02}[flow]
    p0 = {"blast": 0.1, "turb": 0.6, "heat": 1.0}[flow]
    wv = _Waves(g, dims, 2 if kmax > 3 else 1, kmax)
    dirs = []
    for k in wv.k:  # solenoidal velocity: mode amplitudes normal to k
        d = [float(v) for v in torch.randn((3,), generator=g)]
        kk, kd = sum(v * v for v in k), sum(a * b for a, b in zip(k, d))
        dirs.append([d[c] - k[c] * kd / kk for c in range(3)])
    for c, v in enumerate((VX, VY, VZ)):
        prim[v] = vamp / math.sqrt(3.0) * wv.at(xc, yc, zc, [d[c] for d in dirs])
    prim[RHO] = torch.exp(0.05 * scal()) if flow != "heat" else 1.0
    prim[PSC] = 0.5 + 0.2 * torch.tanh(scal())
    if flow == "heat":
        prim[PR] = torch.clamp(1.0 + 0.5 * scal(), min=0.2)
    else:
        prim[PR] = p0 * torch.exp(0.05 * scal())
    if flow == "blast":
        c = [u(0.3, 0.7) for _ in range(3)]
        r2 = (xc - c[0])[None, None, :] ** 2 + (yc - c[1])[None, :, None] ** 2
        if dims == 3:
            r2 = r2 + (zc - c[2])[:, None, None] ** 2
        prim[PR] = prim[PR] * torch.where(r2 < 0.01, u(10.0, 100.0), 1.0)
    bmag = {"blast": u(0.5, 2.0) / math.sqrt(4 * math.pi), "turb": math.sqrt(2 * p0), "heat": math.sqrt(0.02)}[flow]
    ang = u(0, 2 * math.pi) if flow == "blast" else 0.0
    b0 = (bmag * math.cos(ang), bmag * math.sin(ang), 0.1 * bmag)
    pert = {"blast": 0.02, "turb": 0.3, "heat": 0.1}[flow] * bmag / (2 * math.pi * (2 if kmax > 3 else 1))
    az = pert * _Waves(g, dims, 2 if kmax > 3 else 1, kmax).at(xf, yf, zc)
    bx = torch.diff(az, dim=1) * ny
    by = -torch.diff(az, dim=2) * nx
    bz = torch.zeros((nz + (dims == 3), ny, nx), dtype=F64, device=dev)
    if dims == 3:
        ax = pert * _Waves(g, dims, 2 if kmax > 3 else 1, kmax).at(xc, yf, zf)
        ay = pert * _Waves(g, dims, 2 if kmax > 3 else 1, kmax).at(xf, yc, zf)
        bx = bx - torch.diff(ay, dim=0) * nz
        by = by + torch.diff(ax, dim=0) * nz
        bz = bz + torch.diff(ay, dim=2) * nx - torch.diff(ax, dim=1) * ny
    else:
        bz = bz + 0.05 * bmag * scal()
    return prim, (bx + b0[0], by + b0[1], bz + b0[2])


def _full(case, n, seed, inst, dev="cuda"):
    """_initial on the full arrays (9 | 3, Nz, Ny, Nx), ghosts zero."""
    prim, b = _initial(case, n, seed, inst, dev)
    ng, d3 = 3, n[2] > 1
    shape = (n[2] + 2 * ng if d3 else 1, n[1] + 2 * ng, n[0] + 2 * ng)
    P = torch.zeros((9,) + shape, dtype=F64, device=dev)
    B = torch.zeros((3,) + shape, dtype=F64, device=dev)
    k, j, i = (slice(ng, ng + n[2]) if d3 else slice(0, 1)), slice(ng, ng + n[1]), slice(ng, ng + n[0])
    P[:, k, j, i] = prim
    if not case.get("hydro"):
        B[0, k, j, ng:ng + n[0] + 1] = b[0]
        B[1, k, ng:ng + n[1] + 1, i] = b[1]
        B[2, (slice(ng, ng + n[2] + 1) if d3 else k), j, i] = b[2]
    return P, B


def _rows(case, seed, dev="cuda"):
    """Left and right face states and the normal field of n interfaces."""
    n, g = case["n"], torch.Generator(device=dev)
    g.manual_seed(seed * 7919 + case["n"])
    r = lambda: torch.randn((n,), generator=g, dtype=F64, device=dev)
    w = []
    for _ in range(2):
        v = [torch.exp(0.5 * r()), r(), r(), r(), torch.exp(0.7 * r()), 0.5 + 0.1 * r(), r(), r(), r()]
        w.append(torch.stack(v[:case["nvar"]]))
    bx = r()
    if case["nvar"] == 9:
        w[0][BX] = bx
        w[1][BX] = bx
    return w[0], w[1], bx if case["nvar"] == 9 else None


def prepare(case, seed):
    if case["kind"] == "riemann":
        return dict(case=case, rows=_rows(case, seed))
    sides = _sides(case)
    grids = [dict(Nx=n[0], Ny=n[1], Nz=n[2], dims=_dims(case), bc=_bc(case)) for n in sides]
    st = dict(case=case)
    if case["kind"] in ("sweep", "host"):
        st["batch"] = _lib.Batch(grids, path="fused", **_method(case))
        ctxs = st["batch"].instances
    else:
        ctxs = [_lib.Context(path="split" if _split(case) else "fused", **grids[0], **_method(case))]
    cells = [math.prod(c.shape) for c in ctxs]
    host = case["kind"] == "host"
    flat = lambda nf: torch.zeros(nf * sum(cells), dtype=F64, device="cuda")
    views = lambda f, nf: [t.view((nf,) + c.shape) for t, c in zip(f.split([nf * m for m in cells]), ctxs)]
    prim, bfld, prim_out, bfld_out = flat(9), flat(3), flat(9), flat(3)
    p0, b0 = views(prim, 9), views(bfld, 3)
    for q, (c, n) in enumerate(zip(ctxs, sides)):
        P, B = _full(case, n, seed, q)
        torch.cuda.synchronize()
        c.set_state_device(P.data_ptr(), B.data_ptr())
        c.init()  # ghosts and cell B from the faces
        c.get_state_device(p0[q].data_ptr(), b0[q].data_ptr())
        c.sync()
    st.update(ctxs=ctxs, p0=p0, b0=b0)
    if host:
        # one pinned allocation, each grid's prim then its face field
        buf = torch.empty(12 * sum(cells), dtype=F64, pin_memory=True)
        st["host"], off = [], 0
        for q, m in enumerate(cells):
            hp = buf[off:off + 9 * m].view_as(p0[q]).copy_(p0[q])
            hb = buf[off + 9 * m:off + 12 * m].view_as(b0[q]).copy_(b0[q])
            st["host"].append((hp.numpy(), hb.numpy()))
            off += 12 * m
        st["buf"] = buf
    elif case["kind"] == "rollout":
        st["prim"] = p0[0].clone().requires_grad_()
        st["bfld"] = b0[0].clone().requires_grad_()
        st["target"] = torch.ones_like(p0[0][RHO])
    else:
        st.update(out=(prim_out, bfld_out), po=views(prim_out, 9), bo=views(bfld_out, 3))
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "riemann":
        return _lib.riemann(case["rsolver"], *st["rows"], GAM)
    if case["kind"] == "host":
        st["batch"].step_host([h[0] for h in st["host"]], [h[1] for h in st["host"]])
        return st["buf"]
    if case["kind"] == "rollout":
        prim, bfld = st["prim"], st["bfld"]
        pT, bT = rollout(prim, bfld, st["ctxs"][0], case["steps"], case["dt"], case["every"])
        loss = ((pT[RHO] - st["target"]) ** 2).sum()
        gp, gb = torch.autograd.grad(loss, (prim, bfld))
        return dict(prim=pT.detach(), bfld=bT.detach(), loss=loss.detach(), gprim=gp, gbfld=gb)
    for c, p, b in zip(st["ctxs"], st["p0"], st["b0"]):
        c.set_state_device(p.data_ptr(), b.data_ptr())
    if case["kind"] == "sweep":
        st["batch"].advance(1e30, case["steps"])
    elif case["graph"]:
        st["ctxs"][0].advance_graph(1e30, case["steps"])
    else:
        st["ctxs"][0].advance(1e30, case["steps"])
    for c, p, b in zip(st["ctxs"], st["po"], st["bo"]):
        c.get_state_device(p.data_ptr(), b.data_ptr())
    return dict(prim=st["out"][0], bfld=st["out"][1])


def work(case):
    """Bytes: every step reads the conserved state and the faces once and
    writes them once (192 B a zone), a conduction stage 96 B, a rollout's
    reverse step the recorded and the cotangent state; flops: the FP64
    arithmetic of a zone-update."""
    if case["kind"] == "riemann":
        return {"bytes": 8.0 * case["n"] * (3 * case["nvar"] + (case["nvar"] == 9)), "flops": 350.0 * case["n"]}
    zones = float(sum(n[0] * n[1] * n[2] for n in _sides(case)))
    dims = _dims(case)
    zu = zones * case["steps"]
    flops = 450.0 * 2 * dims * zu
    if case["kind"] == "rollout":
        return {"bytes": 192.0 * 3 * zu, "flops": 3 * flops}
    b = 192.0 * zu
    if case.get("kappa0"):
        b += 4 * 96.0 * zu
    if case["kind"] == "host":
        b += 2 * 96.0 * zones
    return {"bytes": b, "flops": flops}


def tolerance(case):
    """FP64 throughout.  Against exact() the steps are off by up to 2e-15 (2-norm)
    and 3e-13 (largest), the gradient of 100 steps by 3e-10 and 1e-8 (limiters and
    wave speeds close to a switch); about four times that with a margin for other
    draws and states."""
    if case["kind"] == "rollout":
        return {"rel": 2e-9, "max": 2e-7}
    if case["kind"] == "riemann":  # strong random states; hllt divides by near-cancelling speeds
        return {"rel": 3e-14, "max": 2e-11}
    return {"rel": 2e-14, "max": 4e-12}


# ---------------------------------------------------------------------------
# the same work in plain torch, FP64
# ---------------------------------------------------------------------------

def _sqr(x):
    return x * x


def _prim2cons(w):
    v2 = _sqr(w[VX]) + _sqr(w[VY]) + _sqr(w[VZ])
    b2 = _sqr(w[BX]) + _sqr(w[BY]) + _sqr(w[BZ])
    return [w[RHO], w[RHO] * w[VX], w[RHO] * w[VY], w[RHO] * w[VZ], 0.5 * (w[RHO] * v2 + b2) + w[PR] / (GAM - 1),
            w[PSC], w[BX], w[BY], w[BZ]]


def _cons2prim(u):
    v = [u[1] / u[0], u[2] / u[0], u[3] / u[0]]
    ke = 0.5 * u[0] * (_sqr(v[0]) + _sqr(v[1]) + _sqr(v[2]))
    me = 0.5 * (_sqr(u[BX]) + _sqr(u[BY]) + _sqr(u[BZ]))
    return [u[0], v[0], v[1], v[2], (GAM - 1) * (u[4] - ke - me), u[5], u[BX], u[BY], u[BZ]]


def _flux(w, u):
    """Physical flux along the local x of a state (the normal field's is zero)."""
    b2 = _sqr(w[BX]) + _sqr(w[BY]) + _sqr(w[BZ])
    vb = w[VX] * w[BX] + w[VY] * w[BY] + w[VZ] * w[BZ]
    pt = w[PR] + 0.5 * b2
    return [u[0] * w[VX], u[1] * w[VX] + pt - _sqr(w[BX]), u[2] * w[VX] - w[BX] * w[BY],
            u[3] * w[VX] - w[BX] * w[BZ], (u[4] + pt) * w[VX] - w[BX] * vb, u[5] * w[VX], torch.zeros_like(w[RHO]),
            w[VX] * w[BY] - w[VY] * w[BX], w[VX] * w[BZ] - w[VZ] * w[BX]]


def _fast(w):
    gp = GAM * w[PR]
    c1 = gp + _sqr(w[BX]) + _sqr(w[BY]) + _sqr(w[BZ])
    return torch.sqrt(0.5 / w[RHO] * (c1 + torch.sqrt(torch.abs(c1 * c1 - 4 * gp * _sqr(w[BX])))))


def _hll(L, R):
    uL, uR = _prim2cons(L), _prim2cons(R)
    fL, fR = _flux(L, uL), _flux(R, uR)
    cf = torch.maximum(_fast(L), _fast(R))
    aL = torch.clamp(torch.minimum(L[VX], R[VX]) - cf, max=0.0)
    aR = torch.clamp(torch.maximum(L[VX], R[VX]) + cf, min=0.0)
    f = [(aR * fL[n] - aL * fR[n] + aL * aR * (uR[n] - uL[n])) / (aR - aL) for n in range(9)]
    f[BX] = torch.zeros_like(f[0])
    return f


def _hllc(L, R):
    """Toro's HLLC with pressure-based wave speeds (no field)."""
    aL, aR = torch.sqrt(GAM * L[PR] / L[RHO]), torch.sqrt(GAM * R[PR] / R[RHO])
    pv = torch.clamp(0.5 * (L[PR] + R[PR]) - 0.125 * (R[VX] - L[VX]) * (L[RHO] + R[RHO]) * (aL + aR), min=0.0)
    q = lambda p: torch.where(pv < p, torch.ones_like(p),
                              torch.sqrt(1 + 0.5 * (GAM + 1) / GAM * (torch.clamp(pv / p, min=1.0) - 1)))
    sL, sR = L[VX] - aL * q(L[PR]), R[VX] + aR * q(R[PR])
    xL, xR = L[RHO] * (L[VX] - sL), R[RHO] * (R[VX] - sR)
    yL, yR = L[PR] + L[RHO] * L[VX] * (L[VX] - sL), R[PR] + R[RHO] * R[VX] * (R[VX] - sR)
    sM = (yR - yL) / (xR - xL)
    ps = (xR * yL - xL * yR) / (xR - xL)
    left = sM > 0
    w = [torch.where(left, a, b) for a, b in zip(L, R)]
    s = torch.where(left, torch.clamp(sL, max=0.0), torch.clamp(sR, min=0.0))
    u = _prim2cons(w)
    f = [u[n] * (w[VX] - s) for n in range(6)]
    f[1] = f[1] + w[PR]
    f[4] = f[4] + w[PR] * w[VX]
    z, t = -sM / (s - sM), s / (s - sM) * ps
    f = [z * v for v in f]
    f[1] = f[1] + t
    f[4] = f[4] + t * sM
    return f + [torch.zeros_like(sM)] * 3


def _hll_hydro(L, R):
    uL, uR = _prim2cons(L), _prim2cons(R)
    fL, fR = _flux(L, uL), _flux(R, uR)
    cf = torch.maximum(torch.sqrt(GAM * L[PR] / L[RHO]), torch.sqrt(GAM * R[PR] / R[RHO]))
    aL = torch.clamp(torch.minimum(L[VX], R[VX]) - cf, max=0.0)
    aR = torch.clamp(torch.maximum(L[VX], R[VX]) + cf, min=0.0)
    f = [(aR * fL[n] - aL * fR[n] + aL * aR * (uR[n] - uL[n])) / (aR - aL) for n in range(6)]
    return f + [torch.zeros_like(f[0])] * 3


def _hllt(L, R):
    """Three-wave solver whose star states carry no energy."""
    uL, uR = _prim2cons(L), _prim2cons(R)
    fL, fR = _flux(L, uL), _flux(R, uR)
    cf = torch.maximum(_fast(L), _fast(R))
    sL, sR = torch.minimum(L[VX], R[VX]) - cf, torch.maximum(L[VX], R[VX]) + cf
    bx, d = L[BX], sR - sL
    star = lambda n: (sR * uR[n] - sL * uL[n] - (fR[n] - fL[n])) / d
    rs, ms, cs = star(0), star(1), star(5)
    us = (sR * fL[0] - sL * fR[0] + sR * sL * (uR[0] - uL[0])) / d / rs
    ca = torch.abs(bx) / torch.sqrt(rs)
    sLs, sRs, zero = us - ca, us + ca, torch.zeros_like(rs)
    S = []
    for w, s in ((L, sL), (R, sR)):
        x = 1 / ((s - sLs) * (s - sRs))
        y, h = bx * x * (us - w[VX]), (w[RHO] * _sqr(s - w[VX]) - _sqr(bx)) / rs * x
        S.append([rs, ms, rs * w[VY] - y * w[BY], rs * w[VZ] - y * w[BZ], zero, cs, zero, h * w[BY], h * w[BZ]])
    x = 0.5 * torch.sign(bx) * torch.sqrt(rs)
    a, b = S
    C = [rs, ms, 0.5 * (a[2] + b[2]) + x * (b[BY] - a[BY]), 0.5 * (a[3] + b[3]) + x * (b[BZ] - a[BZ]), zero, cs, zero,
         0.5 * (a[BY] + b[BY]) + x / rs * (b[2] - a[2]), 0.5 * (a[BZ] + b[BZ]) + x / rs * (b[3] - a[3])]
    out = []
    for n in range(9):
        l1 = fL[n] + sL * (a[n] - uL[n])
        v = torch.where(sL > 0, fL[n], l1)
        v = torch.where((sLs <= 0) & (sRs > 0), l1 + sLs * (C[n] - a[n]), v)
        v = torch.where(sRs <= 0, fR[n] + sR * (b[n] - uR[n]), v)
        out.append(torch.where(sR <= 0, fR[n], v))
    out[BX] = zero
    return out


def _hlld(L, R):
    """Miyoshi & Kusano (2005)."""
    bx = L[BX]
    bx2, sg = _sqr(bx), torch.sign(bx)
    uL, uR = _prim2cons(L), _prim2cons(R)
    fL, fR = _flux(L, uL), _flux(R, uR)
    cf = torch.maximum(_fast(L), _fast(R))
    sL, sR = torch.minimum(L[VX], R[VX]) - cf, torch.maximum(L[VX], R[VX]) + cf
    sM = (sR * uR[1] - sL * uL[1] - (fR[1] - fL[1])) / (sR * uR[0] - sL * uL[0] - (fR[0] - fL[0]))
    pt = lambda w: w[PR] + 0.5 * (bx2 + _sqr(w[BY]) + _sqr(w[BZ]))
    ps = L[RHO] * (sL - L[VX]) * (sM - L[VX]) + pt(L)
    S = []
    for w, u, s in ((L, uL, sL), (R, uR, sR)):
        sv = s - w[VX]
        x = sv / (s - sM)
        den = w[RHO] * sv * (s - sM) - bx2
        f, h = bx * (sM - w[VX]) / den, (w[RHO] * sv * sv - bx2) / den
        vy, vz, by, bz = w[VY] - w[BY] * f, w[VZ] - w[BZ] * f, w[BY] * h, w[BZ] * h
        vb = sM * bx + vy * by + vz * bz
        e = (sv * u[4] - pt(w) * w[VX] + ps * sM + bx * (w[VX] * bx + w[VY] * w[BY] + w[VZ] * w[BZ] - vb)) / (s - sM)
        S.append((w[RHO] * x, vy, vz, by, bz, vb, e, u[5] * x))
    (rL, vyL, vzL, byL, bzL, vbL, eL, cL), (rR, vyR, vzR, byR, bzR, vbR, eR, cR) = S
    qL, qR = torch.sqrt(rL), torch.sqrt(rR)
    sLs, sRs = sM - torch.abs(bx) / qL, sM + torch.abs(bx) / qR
    vyd = (qL * vyL + qR * vyR + (byR - byL) * sg) / (qL + qR)
    vzd = (qL * vzL + qR * vzR + (bzR - bzL) * sg) / (qL + qR)
    byd = (qL * byR + qR * byL + qL * qR * (vyR - vyL) * sg) / (qL + qR)
    bzd = (qL * bzR + qR * bzL + qL * qR * (vzR - vzL) * sg) / (qL + qR)
    vbd = sM * bx + vyd * byd + vzd * bzd
    zero = torch.zeros_like(sM)
    us = lambda r, vy, vz, by, bz, e, c: [r, r * sM, r * vy, r * vz, e, c, zero, by, bz]
    aL, aR = us(rL, vyL, vzL, byL, bzL, eL, cL), us(rR, vyR, vzR, byR, bzR, eR, cR)
    dL = us(rL, vyd, vzd, byd, bzd, eL - qL * (vbL - vbd) * sg, cL)
    dR = us(rR, vyd, vzd, byd, bzd, eR + qR * (vbR - vbd) * sg, cR)
    out = []
    for n in range(9):
        l1, r1 = fL[n] + sL * (aL[n] - uL[n]), fR[n] + sR * (aR[n] - uR[n])
        v = torch.where(sL > 0, fL[n], l1)
        v = torch.where((sLs <= 0) & (sM > 0), l1 + sLs * (dL[n] - aL[n]), v)
        v = torch.where((sM <= 0) & (sRs > 0), r1 + sRs * (dR[n] - aR[n]), v)
        v = torch.where((sRs <= 0) & (sR > 0), r1, v)
        out.append(torch.where(sR <= 0, fR[n], v))
    out[BX] = zero
    return out


def _solver(case):
    if case.get("hydro") or case.get("nvar") == 6:
        return _hllc if case["rsolver"] == "hllc" else _hll_hydro
    return {"hll": _hll, "hllt": _hllt, "hlld": _hlld}[case["rsolver"]]


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(torch.abs(a) < torch.abs(b), a, b))


def _limit(lim, a, b):
    if lim == "mm":
        return _minmod(a, b)
    if lim == "mc":
        return _minmod(2 * _minmod(a, b), 0.5 * (a + b))
    ab = a * b
    up = ab > 0
    return torch.where(up, 2 * ab / torch.where(up, a + b, torch.ones_like(a)), torch.zeros_like(a))


def _char_slopes(lim, dm, dp, w):
    """Limited differences in the characteristic variables of the state w
    (Stone et al. 2008 eigenvectors); the scalar and the normal field pass through."""
    rho, s = w[RHO], torch.sign(w[BX])
    a2r, bp2 = GAM * w[PR], _sqr(w[BY]) + _sqr(w[BZ])
    x = a2r + _sqr(w[BX]) + bp2
    y = torch.sqrt(torch.abs(x * x - 4 * a2r * _sqr(w[BX])))
    f2, s2 = 0.5 * (x + y), 0.5 * (x - y)
    a, cf, cs = torch.sqrt(a2r / rho), torch.sqrt(f2 / rho), torch.sqrt(torch.abs(s2) / rho)
    one, zero = torch.ones_like(rho), torch.zeros_like(rho)
    lo, mid, hi = cf <= cs, a <= cs, cf <= a
    af = torch.where(lo, one, torch.where(mid, zero, torch.where(hi, one, torch.sqrt(torch.abs(a2r - s2) / (f2 - s2)))))
    az = torch.where(lo, zero, torch.where(mid, one, torch.where(hi, zero, torch.sqrt(torch.abs(f2 - a2r) / (f2 - s2)))))
    nz = bp2 != 0
    bt = torch.sqrt(torch.where(nz, bp2, one))
    ty, tz = torch.where(nz, w[BY] / bt, zero), torch.where(nz, w[BZ] / bt, zero)
    nf, sr = 0.5 / (a2r / rho), torch.sqrt(rho)

    def project(d):
        v, b = ty * d[VY] + tz * d[VZ], ty * d[BY] + tz * d[BZ]
        t = lambda p, q: p * (-tz * d[VY] + ty * d[VZ]) + s / sr * (-tz * d[BY] + ty * d[BZ]) * q
        pr = d[PR] / rho
        fast = lambda g: nf * (af * (pr + g * cf * d[VX]) - g * cs * az * s * v + az * a / sr * b)
        slow = lambda g: nf * (az * (pr + g * cs * d[VX]) + g * cf * af * s * v - af * a / sr * b)
        return [fast(-1), 0.5 * t(1, 1), slow(-1), d[RHO] - 2 * nf * d[PR], slow(1), d[PSC], d[BX], 0.5 * t(-1, 1),
                fast(1)]

    m, p = project(dm), project(dp)
    c = [_limit(lim, u, v) for u, v in zip(m, p)]
    e = af * (c[0] + c[8]) + az * (c[2] + c[4])
    t = cs * az * s * (c[0] - c[8]) - cf * af * s * (c[2] - c[4])
    u = a * sr * (az * (c[0] + c[8]) - af * (c[2] + c[4]))
    k, q = c[1] - c[7], s * sr * (c[1] + c[7])
    return [rho * e + c[3], cf * af * (c[8] - c[0]) + cs * az * (c[4] - c[2]), ty * t - tz * k, tz * t + ty * k,
            a2r * e, c[5], c[6], ty * u - tz * q, tz * u + ty * q]


def _perm(ax):
    """Global variable of each local one in the sweep along ax."""
    v, b = [VX, VY, VZ], [BX, BY, BZ]
    v, b = v[ax:] + v[:ax], b[ax:] + b[:ax]
    return [RHO] + v + [PR, PSC] + b


def _dn(a, ax):
    """The value at the index below along axis ax (x = 0) of (..., z, y, x)."""
    return torch.roll(a, 1, dims=-1 - ax)


def _up(a, ax):
    return torch.roll(a, -1, dims=-1 - ax)


class _Exact:
    """Steps of one grid on full arrays with ghosts: every stage is formed on
    the whole array by shifts, the cells that a shift spoils lie in the ghosts."""

    def __init__(self, case, n):
        self.case, self.n = case, n
        self.dims = 3 if n[2] > 1 else 2
        self.ng = 3
        self.solver = _solver(case)
        self.bc = (case["bcx"], case["bcy"], case["bcz"])
        self.h = [1.0 / n[d] for d in range(3)]
        ng = self.ng
        self.act = tuple(slice(ng, ng + n[d]) if d < self.dims else slice(0, 1) for d in (2, 1, 0))

    def _map(self, ax, face):
        """Source index and factor of every index along ax (boundary conditions)."""
        n, a1, f = self.n[ax], self.ng, self.bc[ax]
        a2 = a1 + n - 1
        src, fac = [], []
        for q in range(n + 2 * self.ng):
            s, g = q, 1.0
            if f == 0:
                s = a1 + (q - a1) % n
            elif f == 1:
                s = min(max(q, a1), a2 + 1 if face else a2)
            elif face:
                s = 2 * a1 - q if q < a1 else 2 * a2 + 2 - q if q > a2 + 1 else q
                g = 0.0 if q in (a1, a2 + 1) else -1.0 if s != q else 1.0
            else:
                s = 2 * a1 - 1 - q if q < a1 else 2 * a2 + 1 - q if q > a2 else q
                g = -1.0 if s != q else 1.0
            src.append(s)
            fac.append(g)
        return src, fac

    def fill(self, a, normal=None, face=None):
        """One array's ghosts; normal: the axis whose reflection flips its sign."""
        for ax in reversed(range(self.dims)):
            src, fac = self._map(ax, face == ax)
            a = a.index_select(a.dim() - 1 - ax, torch.tensor(src, device=a.device))
            if normal == ax and self.bc[ax] == 2:
                shape = [1, 1, 1]
                shape[2 - ax] = len(fac)
                a = a * torch.tensor(fac, dtype=F64, device=a.device).view(shape)
        return a

    def fill_all(self, W, B):
        normal = {VX: 0, VY: 1, VZ: 2, BX: 0, BY: 1, BZ: 2}
        W = [self.fill(w, normal.get(v) if normal.get(v, 9) < self.dims else None) for v, w in enumerate(W)]
        B = [self.fill(b, d, d) if d < self.dims else self.fill(b) for d, b in enumerate(B)]
        return W, B

    def start(self, P, B):
        """Ghosts and cell fields of an initial state (active cells and faces)."""
        W, B = self.fill_all(list(P), list(B))
        W[BX:] = self.cell_b(B)
        return self.fill_all(W, B)

    def cell_b(self, B):
        return [0.5 * (B[d] + _up(B[d], d)) if d < self.dims else B[d] for d in range(3)]

    def stage(self, Wf, Bf, Wn, Bn, dt, plm):
        c, D = self.case, self.dims
        F = []
        for ax in range(D):
            p = _perm(ax)
            w = [Wf[v] for v in p]
            if plm:
                dm = [v - _dn(v, ax) for v in w]
                dp = [_up(v, ax) - v for v in w]
                if c["charact"]:
                    d = _char_slopes(c["limiter"], dm, dp, w)
                else:
                    d = [_limit(c["limiter"], a, b) for a, b in zip(dm, dp)]
                L = [_dn(v + 0.5 * s, ax) for v, s in zip(w, d)]
                R = [v - 0.5 * s for v, s in zip(w, d)]
            else:
                L, R = [_dn(v, ax) for v in w], w[:]
            L[BX] = R[BX] = Bf[ax]
            f = self.solver(L, R)
            F.append({v: f[q] for q, v in enumerate(p)})
        u = _prim2cons(Wn)
        for ax in range(D):
            for v in range(6):
                u[v] = u[v] - dt / self.h[ax] * (_up(F[ax][v], ax) - F[ax][v])
        B = list(Bn)
        if not c.get("hydro"):
            v, b = Wf[VX:VZ + 1], Wf[BX:]
            ec = [v[2] * b[1] - v[1] * b[2], v[0] * b[2] - v[2] * b[0], v[1] * b[0] - v[0] * b[1]]
            x, y = F[0], F[1]

            def edge(fa, fb, e, p, q):  # flux sums of two directions and the four cells' fields
                g = e + _dn(e, p)
                return 0.5 * (fa + fb) - 0.25 * (g + _dn(g, q))

            both = lambda a, ax: a + _dn(a, ax)
            E2 = edge(-both(x[BY], 1), both(y[BX], 0), ec[2], 0, 1)
            if D == 3:
                z = F[2]
                E0 = edge(-both(y[BZ], 2), both(z[BY], 1), ec[0], 1, 2)
                E1 = edge(-both(z[BX], 0), both(x[BZ], 2), ec[1], 0, 2)
            else:
                E0, E1 = -y[BZ], x[BZ]
            dd = lambda e, ax: dt / self.h[ax] * (_up(e, ax) - e)
            B[0] = Bn[0] - dd(E2, 1)
            B[1] = Bn[1] + dd(E2, 0)
            B[2] = Bn[2] - dd(E1, 0) + dd(E0, 1)
            if D == 3:
                B[0] = B[0] + dd(E1, 2)
                B[1] = B[1] - dd(E0, 2)
        u[BX:] = self.cell_b(B)
        if c["grav"]:
            u[2] = u[2] + dt * c["grav"] * Wf[RHO]
            u[4] = u[4] + dt * c["grav"] * Wf[RHO] * Wf[VY]
        return _cons2prim(u), B

    def cfl(self, W):
        w = [v[self.act] for v in W]
        cf = torch.sqrt(GAM * w[PR] / w[RHO]) if self.case.get("hydro") else _fast(w)
        m = max(float(((torch.abs(w[VX + d]) + cf) / self.h[d]).max()) for d in range(self.dims))
        return (0.3 if self.dims == 3 else 0.4) / m

    def step(self, W, B, dt):
        Ws, Bs = self.stage(W, B, W, B, 0.5 * dt, False)
        W, B = self.stage(Ws, Bs, W, B, dt, True)
        W, B = self.fill_all(W, B)
        if self.case.get("kappa0"):
            W = self.conduct(W, B, dt)
        return W, B

    def heat(self, p, W, B):
        """-(gamma - 1) div q of the field-aligned flux with limited transverse gradients."""
        T = p / W[RHO]

        def lim(a, b):
            a, b = torch.abs(a), torch.abs(b)
            return torch.minimum(torch.minimum(0.5 * (a + b), a), b)

        g = [(T - _dn(T, d)) / self.h[d] for d in range(3)]
        tr = [lim(g[d], _up(g[d], d)) for d in range(3)]
        out = 0.0
        for ax in range(3):
            b = [B[d] if d == ax else 0.5 * (W[BX + d] + _dn(W[BX + d], ax)) for d in range(3)]
            inv = 1 / torch.sqrt(_sqr(b[0]) + _sqr(b[1]) + _sqr(b[2]) + 1e-20)
            grad = [g[d] if d == ax else lim(_dn(tr[d], ax), tr[d]) for d in range(3)]
            q = -self.case["kappa0"] * b[ax] * inv * sum(b[d] * inv * grad[d] for d in range(3))
            out = out - (GAM - 1) * (_up(q, ax) - q) / self.h[ax]
        return out

    def conduct(self, W, B, dt):
        """RKL2 super-time-stepping (Meyer et al. 2014) of the pressure."""
        k = self.case["kappa0"]
        mx = float((k / W[RHO][self.act] * (GAM - 1)).max()) * sum(1 / h ** 2 for h in self.h)
        dd = 0.5 / mx
        s = 1 if dd >= dt else int(0.5 * (math.sqrt(9 + 16 * dt / dd) - 1)) + 1
        p0 = W[PR]
        M0 = self.heat(p0, W, B)
        if s == 1:
            p = p0 + dt * M0
        else:
            b = [1 / 3.0] * 2 + [(j * j + j - 2) / (2.0 * j * (j + 1)) for j in range(2, s + 1)]
            w1 = 4.0 / (s * s + s - 2)
            prev, p = p0, self.fill(p0 + dt * w1 * b[1] * M0)
            for j in range(2, s + 1):
                mu, nu = (2.0 * j - 1) / j * b[j] / b[j - 1], (1.0 - j) / j * b[j] / b[j - 2]
                q = (mu * p + nu * prev + (1 - mu - nu) * p0 +
                     dt * w1 * mu * (self.heat(p, W, B) + (b[j - 1] - 1) * M0))
                prev, p = p, self.fill(q)
        W = list(W)
        W[PR] = self.fill(p)
        return W


def _exact_grid(case, n, seed, inst):
    P, B = _full(case, n, seed, inst)
    G = _Exact(case, n)
    W, B = G.start(P, B)
    for _ in range(case["steps"]):
        W, B = G.step(W, B, G.cfl(W))
    return torch.stack(W), torch.stack(B)


def _exact_rollout(case, seed):
    from torch.utils.checkpoint import checkpoint
    n = (case["nx"], case["ny"], 1)
    G = _Exact(case, n)
    W, B = G.start(*_full(case, n, seed, 0))
    prim, bfld = torch.stack(W).requires_grad_(), torch.stack(B).requires_grad_()

    def one(p, b):
        W, B = G.fill_all(list(p), list(b))
        W, B = G.step(W, B, case["dt"])
        return torch.stack(W), torch.stack(B)

    p, b = prim, bfld
    for _ in range(case["steps"]):
        p, b = checkpoint(one, p, b, use_reentrant=False)
    loss = ((p[RHO] - 1.0) ** 2).sum()
    gp, gb = torch.autograd.grad(loss, (prim, bfld))
    return dict(prim=p.detach(), bfld=b.detach(), loss=loss.detach(), gprim=gp, gbfld=gb)


def exact(case, seed):
    if case["kind"] == "riemann":
        wl, wr, bx = _rows(case, seed)
        zero = [torch.zeros_like(wl[0])] * (9 - case["nvar"])
        return torch.stack(_solver(case)(list(wl) + zero, list(wr) + zero)[:case["nvar"]])
    if case["kind"] == "rollout":
        return _exact_rollout(case, seed)
    got = [_exact_grid(case, n, seed, q) for q, n in enumerate(_sides(case))]
    if case["kind"] == "host":
        return torch.cat([t.reshape(-1).cpu() for pb in got for t in pb])
    return dict(prim=torch.cat([p.reshape(-1) for p, _ in got]), bfld=torch.cat([b.reshape(-1) for _, b in got]))
