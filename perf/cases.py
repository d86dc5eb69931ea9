"""The calls whose speed matters to a program that uses this solver library.

Each case is one call (or one step of calls) as a flow solver makes it through
the public interface: Krylov solves on device arrays and through the
Fortran-facing host interface, a batched plan, a differentiable solve, and the
two matrix assemblies.  Matrices are those of perturbed hexahedral boxes with
the coefficients the reference's assembly routines produce (pressure
correction with a smooth variable density, walls and an outlet; first-order
upwind convection and diffusion with a time term); every value and right-hand side comes from the
seed.  Patterns, meshes and solver handles depend on the mesh alone and are
kept between preparations, as a time-stepping program keeps them.

Case keys: ``kind`` ("solve", "legacy", "batch", "adjoint", "calcps",
"newuvw"), the box ``nx, ny, nz``; for solves ``system`` ("pressure" or
"transport"), ``numbering`` ("box": x fastest; "blocks": eight blocks numbered
one after another, as a multi-block mesh generator does), ``method``,
``prec``, ``precision``, ``rtol`` (times ||b||) and ``maxiter``.
"""
import math

import numpy as np
import torch

import __graft_entry__

tf = __graft_entry__.load_package()

DEV = "cuda"
F64 = torch.float64
PRECISION = {"fp64": tf.FP64, "fma": tf.FP64_FMA, "mixed": tf.MIXED}


# ---- the cases -------------------------------------------------------------------

def _solve(name, shape, system, method, prec, precision, rtol, maxiter, numbering="box",
           kind="solve"):
    return {"name": name, "kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2],
            "system": system, "numbering": numbering, "method": method, "prec": prec,
            "precision": precision, "rtol": rtol, "maxiter": maxiter}


def listed():
    return [
        # pressure assembly of a small mesh (one rank's share of a coarse
        # case): microseconds of work, so launches and host calls count
        {"name": "calcps-small", "kind": "calcps", "nx": 48, "ny": 40, "nz": 36, "nmat": 1},
        # the small pressure solve of the 32^3 benchmark: hundreds of short
        # iterations on data that stays in L2
        _solve("pressure-32", (32, 32, 32), "pressure", "cg", 1, "fp64", 1e-8, 20000),
        # species transport from the Fortran program: host arrays in, host
        # arrays out, the default precision, odd mesh sizes
        _solve("species-host", (101, 67, 83), "transport", "cgs", 1, "fp64", 1e-8, 200,
               kind="legacy"),
        # the momentum solve of the 128^3 benchmark: a few iterations, so the
        # set-up of a solve counts as well
        _solve("momentum-128", (128, 128, 128), "transport", "bicg", 1, "fma", 1e-8, 200),
        # differentiable pressure solve: forward and transposed solve, the
        # gradients of the matrix values and the right-hand side
        {"name": "adjoint-64", "kind": "adjoint", "nx": 64, "ny": 64, "nz": 64, "rtol": 1e-10},
        # IC(0) pressure solve on a multi-block mesh, default precision
        _solve("pressure-ic-blocks", (60, 52, 45), "pressure", "cg", 2, "fp64", 1e-11, 2000,
               numbering="blocks"),
        # IC(0) pressure solve on a ragged box, FP64 with multiply-adds
        _solve("pressure-ic-ragged", (109, 83, 97), "pressure", "cg", 2, "fma", 1e-11, 2000),
        # the benchmark's headline solver at 128^3: mixed precision, IC(0)
        # with BF16 factors, to the tolerance of the differentiable solver
        _solve("pressure-mixed-ic", (128, 128, 128), "pressure", "cg", 2, "mixed", 1e-12, 4000),
        # mixed precision with the diagonal on a large ragged box
        _solve("pressure-mixed-diag", (161, 150, 170), "pressure", "cg", 1, "mixed", 1e-12, 8000),
        # one SIMPLE inner solve at the largest size: iterations capped, as
        # the outer loop converges it
        _solve("pressure-256", (256, 256, 256), "pressure", "cg", 1, "fma", 1e-8, 100),
        # independent systems of uneven size in one captured launch
        {"name": "batch-uneven", "kind": "batch", "count": 12, "lo": 16, "hi": 72, "rtol": 1e-12},
        # momentum assembly of the benchmark mesh, blended convection
        {"name": "newuvw-128", "kind": "newuvw", "nx": 128, "ny": 128, "nz": 128, "nmat": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box_shape(rng, lo_cells, hi_cells):
    """A box of about log-uniform volume whose edges differ by up to a third."""
    n = _log_int(rng, lo_cells, hi_cells)
    e = n ** (1.0 / 3.0)
    fx, fy = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    nx, ny = max(4, int(e * fx)), max(4, int(e * fy))
    return nx, ny, max(4, min(n // (nx * ny), int(1.4 * e)))


def draw(rng):
    kind = rng.choice(["solve"] * 7 + ["legacy", "legacy", "batch", "adjoint", "calcps", "newuvw"])
    if kind in ("calcps", "newuvw"):
        nx, ny, nz = _box_shape(rng, 4000, 2_000_000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nmat": rng.choice([1, 1, 2])}
    if kind == "adjoint":
        nx, ny, nz = _box_shape(rng, 4000, 262_144)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "rtol": 1e-10}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 14), "lo": rng.randint(12, 24),
                "hi": rng.randint(40, 72), "rtol": 1e-12}
    system = rng.choice(["pressure", "transport"])
    method = "cg" if system == "pressure" else rng.choice(["bicg", "cgs"])
    prec = rng.choice([1, 2]) if system == "pressure" else 1
    precision = rng.choice(["fp64", "fma", "mixed"]) if kind == "solve" else "fp64"
    numbering = rng.choice(["box", "box", "blocks"])
    if kind == "legacy":
        hi = 60_000 if prec == 2 else 500_000
    elif system == "transport" or (precision == "mixed" and prec == 1):
        hi = 4_000_000
    elif numbering == "blocks" and prec == 2:
        hi = 150_000
    else:
        hi = 1_500_000
    c = _solve("", _box_shape(rng, 4000, hi), system, method, prec, precision,
               1e-12 if precision == "mixed" else 1e-11 if prec == 2 else 1e-8, 8000, numbering,
               kind)
    del c["name"]
    return c


# ---- meshes and systems, made on the device ----------------------------------------

def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(gen, lo, hi, *shape):
    return torch.empty(shape, dtype=F64, device=DEV).uniform_(lo, hi, generator=gen)


def _smooth(gen, shape, sigma):
    """White noise filtered by a periodic Gaussian of `sigma` cells."""
    f = torch.fft.rfftn(torch.randn(shape, dtype=F64, device=DEV, generator=gen))
    for d, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device=DEV) if d == 2 else torch.fft.fftfreq(n, device=DEV)
        g = torch.exp(-2.0 * (math.pi * sigma * k.double()) ** 2)
        f = f * g.reshape([-1 if i == d else 1 for i in range(3)])
    return torch.fft.irfftn(f, s=shape)


def _density(gen, shape):
    f = _smooth(gen, shape, 3.0)
    f = (f - f.min()) / (f.max() - f.min())
    return 0.14 + 0.86 * f


def _dot(a, b):
    return (a * b).sum(0)


def _quads(P):
    """The faces' corner nodes in cyclic order, faces normal to x, y and z."""
    return ((P[:, :-1, :-1, :], P[:, :-1, 1:, :], P[:, 1:, 1:, :], P[:, 1:, :-1, :]),
            (P[:, :-1, :, :-1], P[:, 1:, :, :-1], P[:, 1:, :, 1:], P[:, :-1, :, 1:]),
            (P[:, :, :-1, :-1], P[:, :, :-1, 1:], P[:, :, 1:, 1:], P[:, :, 1:, :-1]))


def _geometry(gen, nx, ny, nz):
    """Nodes displaced by up to 0.2 of the spacing, face area vectors and
    centres per direction, cell centres."""
    z, y, x = torch.meshgrid(*(torch.arange(n + 1, dtype=F64, device=DEV) for n in (nz, ny, nx)),
                             indexing="ij")
    P = torch.stack((x, y, z)) + _uniform(gen, -0.2, 0.2, 3, nz + 1, ny + 1, nx + 1)
    S, Fc = [], []
    for a, b, c, d in _quads(P):
        S.append(0.5 * torch.linalg.cross(c - a, d - b, dim=0))
        Fc.append(0.25 * (a + b + c + d))
    C = 0.5 * (Fc[2][:, :-1] + Fc[2][:, 1:])
    return P, S, Fc, C


def _lo_hi(a, axis):
    """The lower and the upper cell of every interior face normal to `axis`
    (0 = x) of a (..., nz, ny, nx) cell array."""
    d = a.ndim - 1 - axis
    n = a.shape[d]
    return a.narrow(d, 0, n - 1), a.narrow(d, 1, n - 1)


def _interior(S, C, axis):
    """Area vectors and centre distances of the interior faces."""
    d = 3 - axis
    lo, hi = _lo_hi(C, axis)
    return S[axis].narrow(d, 1, S[axis].shape[d] - 2), hi - lo


def _add_faces(A7, axis, off12, off21, d1, d2):
    """One direction's faces into the seven slots (-z, -y, -x, diagonal, +x,
    +y, +z) of a (nz, ny, nx, 7) matrix."""
    lo, hi = _lo_hi(A7.movedim(3, 0), axis)
    lo[4 + axis] -= off12
    hi[2 - axis] -= off21
    lo[3] += d1
    hi[3] += d2


def _pressure(gen, nx, ny, nz):
    P, S, Fc, C = _geometry(gen, nx, ny, nz)
    rho = _density(gen, (nz, ny, nx))
    A7 = torch.zeros(nz, ny, nx, 7, dtype=F64, device=DEV)
    for axis in range(3):
        s, d = _interior(S, C, axis)
        lo, hi = _lo_hi(rho, axis)
        c = _dot(s, s) / _dot(s, d) * (0.5 * (1.0 / lo + 1.0 / hi))
        _add_faces(A7, axis, c, c, c, c)
    # the outlet at x-max adds its coefficient to the diagonal; walls elsewhere
    s, d = S[0][..., -1], Fc[0][..., -1] - C[..., -1]
    A7[:, :, -1, 3] += _dot(s, s) / _dot(s, d) / rho[:, :, -1]
    b = _uniform(gen, -1.0, 1.0, nz, ny, nx)
    return A7, b - b.mean()


def _transport(gen, nx, ny, nz, nu=1e-2, dt=1e-2):
    P, S, Fc, C = _geometry(gen, nx, ny, nz)
    psi = torch.stack([_smooth(gen, tuple(P.shape[1:]), 2.0) for _ in range(3)])
    for d in (1, 2, 3):  # no flow through the walls
        psi.select(d, 0).zero_()
        psi.select(d, -1).zero_()
    flux, ssum, count = [], 0.0, 0
    for axis, (corners, pots) in enumerate(zip(_quads(P), _quads(psi))):
        f = 0.0
        for k in range(4):
            f = f + 0.5 * _dot(pots[k] + pots[(k + 1) % 4], corners[(k + 1) % 4] - corners[k])
        f = f.narrow(2 - axis, 1, f.shape[2 - axis] - 2)
        s, _ = _interior(S, C, axis)
        ssum, count = ssum + (f * f / _dot(s, s)).sum(), count + f.numel()
        flux.append(f)
    rms = torch.sqrt(ssum / count)
    A7 = torch.zeros(nz, ny, nx, 7, dtype=F64, device=DEV)
    for axis in range(3):
        s, d = _interior(S, C, axis)
        a0 = nu * _dot(s, s) / _dot(s, d)
        f = flux[axis] / rms
        out, inn = f.clamp(min=0.0) + a0, (-f).clamp(min=0.0) + a0
        _add_faces(A7, axis, inn, out, out, inn)
    # walls (about |S|^2 / (S.d) = 2 on a unit mesh) and the time term
    for d in range(3):
        A7[..., 3].select(d, 0).add_(2.0 * nu)
        A7[..., 3].select(d, -1).add_(2.0 * nu)
    u_old = _uniform(gen, -1.0, 1.0, nz, ny, nx)
    A7[..., 3] += 1.0 / dt
    return A7, u_old / dt


_patterns = {}


class _Pattern:
    """Compressed rows of a box mesh: 0-based row pointers, columns and
    diagonal positions, and where each stored entry sits in the seven slots."""

    def __init__(self, nx, ny, nz, numbering):
        n = nx * ny * nz
        cell = torch.arange(n, device=DEV)
        x, y, z = cell % nx, cell // nx % ny, cell // (nx * ny)
        has = torch.stack([z > 0, y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1, z < nz - 1], 1)
        off = torch.tensor([-nx * ny, -nx, -1, 0, 1, nx, nx * ny], device=DEV)
        new = cell
        if numbering == "blocks":
            block = (x >= nx * 2 // 5).long() + 2 * (y >= ny // 2).long() + 4 * (z >= nz // 3).long()
            self.order = torch.argsort(block * n + cell)  # old cell of each new row
            new = torch.empty_like(cell)
            new[self.order] = cell
        else:
            self.order = None
        slot = has.reshape(-1).nonzero()[:, 0]
        row = new[slot // 7]
        col = new[slot // 7 + off[slot % 7]]
        if numbering == "blocks":
            key = torch.argsort(row * n + col)
            slot, row, col = slot[key], row[key], col[key]
        self.n, self.nnz = n, int(slot.numel())
        self.slot = slot
        self.rowptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
        self.rowptr[1:] = torch.bincount(row, minlength=n).cumsum(0)
        self.col = col.to(torch.int32)
        self.diag = (row == col).nonzero()[:, 0].to(torch.int32)
        self.topo = tf.Topology(n, self.rowptr, self.col, self.diag)
        self.solver = None
        self.host = None

    def values(self, A7, b):
        b = b.reshape(-1)
        return A7.reshape(-1)[self.slot], (b if self.order is None else b[self.order]).contiguous()

    def matrix(self, val):
        return torch.sparse_csr_tensor(self.rowptr, self.col, val, (self.n, self.n))

    def fortran(self):
        """1-based host arrays of the layout, as the Fortran program holds them."""
        if self.host is None:
            self.host = tuple(a.cpu().numpy() + 1 for a in (self.rowptr, self.col, self.diag))
            acol, arow, adia = self.host
            self.host = (acol, np.append(arow, np.int32(0)), adia)
        return self.host


def _pattern(nx, ny, nz, numbering="box"):
    key = (nx, ny, nz, numbering)
    if key not in _patterns:
        _patterns[key] = _Pattern(*key)
    return _patterns[key]


def _boundary_cells(case):
    return 2 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nz"] * case["nx"])


def _system(case, seed):
    p = _pattern(case["nx"], case["ny"], case["nz"], case["numbering"])
    make = _pressure if case["system"] == "pressure" else _transport
    return (p, *p.values(*make(_rng(seed), case["nx"], case["ny"], case["nz"])))


# ---- batches ------------------------------------------------------------------------

def _batch_shapes(case):
    """Sizes spread evenly over the logarithm of the cell count, small and
    large ones mixed."""
    k, lo, hi = case["count"], case["lo"], case["hi"]
    out = []
    for j in range(k):
        e = lo * (hi / lo) ** (((j * 5) % k + 0.5) / k)
        n = int(e)
        out.append((n, n, max(4, int(round(e ** 3 / (n * n))))))
    return out


def _batch_systems(case, seed):
    """Odd systems: pressure, CG + IC(0); even ones: transport, BiCG + diagonal."""
    got = []
    for j, shape in enumerate(_batch_shapes(case)):
        c = {"nx": shape[0], "ny": shape[1], "nz": shape[2], "numbering": "box",
             "system": "pressure" if j % 2 else "transport"}
        got.append((*_system(c, seed * 64 + j), "cg" if j % 2 else "bicg", 2 if j % 2 else 1))
    return got


# ---- assemblies ----------------------------------------------------------------------

_meshes = {}
INFLOW, WALL, OUTFLOW = 1, 2, 3
GEOM = ("Sx", "Sy", "Sz", "Dx", "Dy", "Dz", "f", "volume")


def _mesh(nx, ny, nz):
    """A perturbed box with an inflow, an outflow and walls: the mesh arrays
    on the device and the assembly handle made of them."""
    key = (nx, ny, nz)
    if key not in _meshes:
        m = tf.mesh.box_faces(nx, ny, nz, perturb=0.2, seed=7)
        types = np.full(m["NbC"] + m["NC"] + 1, WALL, np.int32)
        types[m["NbC"]:] = 0
        types[m["NbC"] - ny * nz:m["NbC"]] = INFLOW          # x-min: cells -1 ..
        types[m["NbC"] - 2 * ny * nz:m["NbC"] - ny * nz] = OUTFLOW
        g = {k: torch.from_numpy(m[k]).to(DEV) for k in GEOM}
        side = torch.from_numpy(m["SideC"]).to(DEV).long()
        g.update(NC=m["NC"], NbC=m["NbC"], NS=m["NS"], NONZ=int(m["Acol"][-1]),
                 k1=side[:, 1] + m["NbC"], k2=side[:, 2] + m["NbC"], c2=side[:, 2],
                 sid=torch.from_numpy(m["SidAij"]).to(DEV).long() - 1,
                 adia=torch.from_numpy(m["Adia"]).to(DEV).long() - 1,
                 type=torch.from_numpy(types).to(DEV),
                 handle=tf.Assembly.from_faces(m, types))
        _meshes[key] = g
    return _meshes[key]


def _calcps_fields(g, gen):
    m = g["NbC"] + g["NC"] + 1
    f = {k: _uniform(gen, 0.5, 1.5, m) for k in ("rho_n", "rho_o", "rho_oo")}
    f.update({k: _uniform(gen, -1.0, 1.0, m) for k in ("u", "v", "w", "p", "px", "py", "pz")})
    f["asave"] = _uniform(gen, 1.0, 2.0, m)
    return f


GRADS = ("duidi", "duidj", "duidk", "dujdi", "dukdi", "dujdj", "dukdk")
MOMENTUM = dict(visc=1e-2, dt=0.01, urf=0.7)


def _newuvw_fields(g, gen, nmat):
    m, ns = g["NbC"] + g["NC"] + 1, g["NS"]
    f = {k: _uniform(gen, 0.5, 1.5, m) for k in ("rho_n", "rho_o", "rho_oo")}
    f.update({k: _uniform(gen, -1.0, 1.0, m)
              for k in ("ui_n", "ui_o", "ui_oo", *GRADS, "pi", "source")})
    f.update({k: _uniform(gen, -1.0, 1.0, ns) for k in ("flux_u", "flux")})
    f["ff"] = g["f"].clone()
    f["material"] = torch.randint(1, nmat + 1, (m,), dtype=torch.int32, device=DEV, generator=gen)
    f["blend"] = torch.full((nmat,), 24, dtype=torch.int32, device=DEV)      # SMART
    f["blend_tem"] = torch.full((nmat,), 10, dtype=torch.int32, device=DEV)  # YES
    f["urfc"] = torch.full((nmat,), 0.9, dtype=F64, device=DEV)
    return f


# ---- prepare and run -------------------------------------------------------------------

def _options(precision, prec):
    return tf.options(precision=PRECISION[precision], tol_mode=tf.TOL_RELATIVE,
                      ic_bf16=int(precision == "mixed" and prec == 2))


def prepare(case, seed):
    kind, gen = case["kind"], _rng(seed)
    st = {"kind": kind, "case": case}
    if kind == "solve":
        p, val, b = _system(case, seed)
        st.update(p=p, val=val, b=b, opts=_options(case["precision"], case["prec"]),
                  x=torch.zeros(p.n, dtype=F64, device=DEV))
    elif kind == "legacy":
        p, val, b = _system(case, seed)
        nb = _boundary_cells(case)
        st.update(p=p, nb=nb, A=np.append(val.cpu().numpy(), 0.0), b=b.cpu().numpy(),
                  Ab=np.zeros(nb), x=np.zeros(nb + p.n + 1), r=np.zeros(p.n),
                  tol=case["rtol"] * float(b.norm()), layout=p.fortran())
    elif kind == "batch":
        sys = _batch_systems(case, seed)
        topos, vals, bs = ([s[0].topo for s in sys], [s[1] for s in sys], [s[2] for s in sys])
        xs = [torch.zeros_like(b) for b in bs]
        opts = tf.options(precision=tf.MIXED, tol_mode=tf.TOL_RELATIVE, ic_bf16=1)
        n = len(sys)
        st.update(xs=xs, plan=tf.Plan(topos, vals, bs, xs, [s[3] for s in sys],
                                      [s[4] for s in sys], [8000] * n, [case["rtol"]] * n, opts))
    elif kind == "adjoint":
        p = _pattern(case["nx"], case["ny"], case["nz"])
        if p.solver is None:
            from tflows_gb300 import autograd
            p.solver = autograd.DifferentiableSolver(p.topo, p.rowptr.cpu().numpy(),
                                                     p.col.cpu().numpy(), rtol=case["rtol"])
        val, b = p.values(*_pressure(gen, case["nx"], case["ny"], case["nz"]))
        st.update(p=p, val=val.requires_grad_(), b=b.requires_grad_(),
                  target=_uniform(gen, -1.0, 1.0, p.n))
    else:
        g = _mesh(case["nx"], case["ny"], case["nz"])
        f = _calcps_fields(g, gen) if kind == "calcps" else _newuvw_fields(g, gen, case["nmat"])
        st.update(g=g, f=f, aval=torch.empty(g["NONZ"], dtype=F64, device=DEV),
                  b=torch.empty(g["NC"], dtype=F64, device=DEV),
                  abou=torch.zeros(g["NbC"], dtype=F64, device=DEV),
                  flux=torch.empty(g["NS"], dtype=F64, device=DEV),
                  asave=torch.empty(g["NC"], dtype=F64, device=DEV))
    return st


def run(st):
    kind, c = st["kind"], st["case"]
    if kind == "solve":
        st["x"].zero_()
        res = st["p"].topo.solve(st["val"], st["b"], st["x"], c["method"], c["prec"], c["maxiter"],
                                 c["rtol"], opts=st["opts"])
        return {"x": st["x"], "status": res["status"]}
    if kind == "legacy":
        p, (acol, arow, adia) = st["p"], st["layout"]
        st["x"][:] = 0.0
        st["r"][:] = st["b"]
        out = getattr(tf, c["method"])(p.n, st["nb"], p.nnz + 1, st["A"], acol, arow, adia,
                                       st["Ab"], st["x"], st["r"], c["prec"], c["maxiter"],
                                       st["tol"])
        return {"x": st["x"], "niter": out.niter, "status": out.status}
    if kind == "batch":
        for x in st["xs"]:
            x.zero_()
        st["plan"].launch()
        return {"xs": st["xs"], "status": [r["status"] for r in st["plan"].results()]}
    if kind == "adjoint":
        st["val"].grad = st["b"].grad = None
        x = st["p"].solver(st["val"], st["b"])
        (0.5 * ((x - st["target"]) ** 2).sum()).backward()
        return {"x": x.detach(), "grad_val": st["val"].grad, "grad_b": st["b"].grad}
    g = st["g"]
    if kind == "calcps":
        g["handle"].calcps(st["f"], st["aval"], st["b"], st["abou"], st["flux"], Nmat=c["nmat"],
                           dt=0.01)
        return {k: st[k] for k in ("aval", "b", "abou", "flux")}
    g["handle"].newuvw(1, st["f"], st["aval"], st["b"], st["abou"], st["asave"], nmat=c["nmat"],
                       **MOMENTUM)
    return {k: st[k] for k in ("aval", "b", "abou", "asave")}


# ---- what a pass cannot do without --------------------------------------------------------

def _nnz(nx, ny, nz):
    return 7 * nx * ny * nz - 2 * (nx * ny + ny * nz + nz * nx)


def _solve_work(nx, ny, nz, system, prec, maxiter):
    """The matrix and the right-hand side read once and x written once; the
    operations of the iterations a solve of this size takes (for pressure
    about nine per cell of the edge with the diagonal and three with IC(0);
    for transport a handful)."""
    n, nnz = nx * ny * nz, _nnz(nx, ny, nz)
    edge = n ** (1.0 / 3.0)
    its = min(maxiter, 7 if system == "transport" else int(9 * edge if prec == 1 else 3 * edge))
    return {"bytes": 12.0 * nnz + 20.0 * n,
            "flops": its * (2.0 * nnz + 12.0 * n + (2.0 * nnz if prec == 2 else 0.0))}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "legacy"):
        return _solve_work(case["nx"], case["ny"], case["nz"], case["system"], case["prec"],
                           case["maxiter"])
    if kind == "batch":
        w = [_solve_work(*s, "pressure" if j % 2 else "transport", 2 if j % 2 else 1, 8000)
             for j, s in enumerate(_batch_shapes(case))]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, nnz, nb = nx * ny * nz, _nnz(nx, ny, nz), 2 * (nx * ny + ny * nz + nz * nx)
    if kind == "adjoint":
        w = _solve_work(nx, ny, nz, "pressure", 1, 20000)
        return {"bytes": 2 * w["bytes"] + 8.0 * nnz, "flops": 2 * w["flops"]}
    ns = (nnz - n) // 2 + nb
    if kind == "calcps":  # geometry and cells per face, 12 cell fields; Aval, b, fluxes
        return {"bytes": ns * 72.0 + (n + nb) * 100.0 + 4.0 * n + 8.0 * (nnz + n + ns),
                "flops": 40.0 * ns + 25.0 * n}
    return {"bytes": ns * 112.0 + (n + nb) * 136.0 + 4.0 * n + 8.0 * (nnz + 2 * n + nb),
            "flops": 110.0 * ns + 60.0 * n}


# ---- the same results in plain 64-bit torch ------------------------------------------------

def _cg(A, d, b, maxiter, rtol):
    """Diagonally preconditioned CG from zero."""
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, rho = z.clone(), r @ z
    stop = rtol * b.norm()
    for k in range(maxiter):
        q = A @ p
        a = rho / (p @ q)
        x += a * p
        r -= a * q
        if k % 16 == 15 and r.norm() < stop:
            break
        z = r / d
        rho, old = r @ z, rho
        p = z + (rho / old) * p
    return x


def _bicgstab(A, d, b, maxiter, rtol):
    x, r = torch.zeros_like(b), b.clone()
    r0, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho = alpha = omega = 1.0
    for _ in range(maxiter):
        new = float(r0 @ r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
        y = p / d
        v = A @ y
        alpha = rho / float(r0 @ v)
        s = r - alpha * v
        z = s / d
        t = A @ z
        omega = float(t @ s) / float(t @ t)
        x += alpha * y + omega * z
        r = s - omega * t
        if r.norm() < rtol * b.norm():
            break
    return x


def _solution(p, val, b, system):
    """A^-1 b, refined until the residual is at rounding level."""
    A, d = p.matrix(val), val[p.diag.long()]
    x = torch.zeros_like(b)
    for _ in range(3):
        r = b - A @ x
        if r.norm() == 0:
            break
        x = x + (_cg(A, d, r, 20000, 1e-9) if system == "pressure"
                 else _bicgstab(A, d, r, 200, 1e-9))
    return x


def _exact_calcps(case, seed):
    g = _mesh(case["nx"], case["ny"], case["nz"])
    f = _calcps_fields(g, _rng(seed))
    k1, k2, c2 = g["k1"], g["k2"], g["c2"]
    inner, t2 = c2 > 0, g["type"][k2]
    thru, out = (t2 == INFLOW) | (t2 == OUTFLOW), t2 == OUTFLOW
    w, S2 = g["f"], g["Sx"] ** 2 + g["Sy"] ** 2 + g["Sz"] ** 2
    sm = S2 / (g["Sx"] * g["Dx"] + g["Sy"] * g["Dy"] + g["Sz"] * g["Dz"])
    va = g["volume"] / f["asave"]
    a12 = torch.where(inner, 0.5 * sm * (va[k1] + va[k2]), torch.where(out, sm * va[k1], 0.0))
    rho = f["rho_n"]
    flux = 0.0
    for s, u in (("Sx", "u"), ("Sy", "v"), ("Sz", "w")):
        flux = flux + (w * rho[k1] * f[u][k1] + (1 - w) * rho[k2] * f[u][k2]) * g[s]
    grad = 0.0
    for s, q in (("Dx", "px"), ("Dy", "py"), ("Dz", "pz")):
        grad = grad + 0.5 * (f[q][k1] + f[q][k2]) * g[s]
    flux = torch.where(inner, flux + a12 * (f["p"][k1] - f["p"][k2]) + a12 * grad,
                       torch.where(thru, flux, 0.0))
    nb, nmat = g["NbC"], case["nmat"]
    n = nb + g["NC"] + 1
    add = lambda i, v: torch.zeros(n, dtype=F64, device=DEV).index_add_(0, i, v)  # noqa: E731
    d = nmat * (add(k1, a12) + add(k2[inner], a12[inner]))
    b = nmat * (add(k2[inner], flux[inner]) - add(k1, flux))
    b = b - nmat * (g["volume"] / 0.01 * (1.5 * rho - 2.0 * f["rho_o"] + 0.5 * f["rho_oo"]))
    b, vol = b[nb + 1:], g["volume"][nb + 1:]
    aval = torch.zeros(g["NONZ"], dtype=F64, device=DEV)
    aval[g["sid"][inner, 0]] = -a12[inner]
    aval[g["sid"][inner, 1]] = -a12[inner]
    aval[g["adia"]] = d[nb + 1:]
    return {"aval": aval, "b": b - (b * vol).sum() / vol.sum(),
            "abou": torch.zeros(nb, dtype=F64, device=DEV), "flux": flux}


def _exact_newuvw(case, seed):
    g = _mesh(case["nx"], case["ny"], case["nz"])
    f = _newuvw_fields(g, _rng(seed), case["nmat"])
    visc, dt, urf = (MOMENTUM[k] for k in ("visc", "dt", "urf"))
    k1, k2, c2, nb = g["k1"], g["k2"], g["c2"], g["NbC"]
    n = nb + g["NC"] + 1
    inner, t2 = c2 > 0, g["type"][k2]
    phi = f["rho_n"] * f["ui_n"]
    hi, lo = phi.clone(), phi.clone()
    for a, o in ((k1[inner], k2[inner]), (k2[inner], k1[inner])):
        hi.scatter_reduce_(0, a, phi[o], "amax")
        lo.scatter_reduce_(0, a, phi[o], "amin")
    # SMART-limited face value
    up = f["flux"] > 0
    C, D = torch.where(up, k1, k2), torch.where(up, k2, k1)
    fj = torch.where(up, 1 - g["f"], g["f"])
    sign = torch.where(up, 1.0, -1.0).to(F64)
    grad = f["duidi"][C] * g["Dx"] + f["duidj"][C] * g["Dy"] + f["duidk"][C] * g["Dz"]
    u = torch.maximum(lo[C], torch.minimum(phi[D] - sign * 2.0 * grad, hi[C]))
    rj = (phi[C] - u) / (phi[D] - phi[C] + 1.0e-16)
    lim = torch.minimum(2.0 * rj, 0.5 * fj * (1 + fj) + 0.5 * fj * (1 - fj) * rj)
    phis = phi[C] + lim.clamp(max=1.0).clamp(min=0.0) * sign * (phi[k2] - phi[k1])
    fu = f["flux_u"]
    conv = fu * phis - fu * torch.where(fu < 0, phi[k2], phi[k1])
    # diffusion
    w = f["ff"]
    at = lambda k: w * f[k][k1] + (1 - w) * f[k][k2]  # noqa: E731
    ii, ij, ik, ji, ki, jj, kk = (at(k) for k in GRADS)
    fex = visc * (4.0 / 3.0 * ii * g["Sx"] + (ij + ji) * g["Sy"] + (ik + ki) * g["Sz"]
                  - 2.0 / 3.0 * (jj + kk) * g["Sx"])
    a0 = visc * ((g["Sx"] ** 2 + g["Sy"] ** 2 + g["Sz"] ** 2)
                 / (g["Sx"] * g["Dx"] + g["Sy"] * g["Dy"] + g["Sz"] * g["Dz"]))
    fim = a0 * (ii * g["Dx"] + ij * g["Dy"] + ik * g["Dz"])
    q12 = a0 / f["rho_n"][k2] - fu.clamp(max=0.0)
    q21 = a0 / f["rho_n"][k1] + fu.clamp(min=0.0)
    wall, out = (t2 == WALL) | (t2 == INFLOW), t2 == OUTFLOW
    side = torch.where(inner, 0.0, torch.where(wall, q12 * phi[k2],
                                               torch.where(out, -fu.clamp(max=0.0) * phi[k2], 0.0)))
    d1 = torch.where(out & ~inner, fu.clamp(min=0.0), q21)
    add = lambda i, v: torch.zeros(n, dtype=F64, device=DEV).index_add_(0, i, v)  # noqa: E731
    x = 0.9 * conv
    b = add(k2[inner], x[inner]) - add(k1, x)
    x = fex - fim
    b = b + add(k1, x) - add(k2[inner], x[inner]) + add(k1, side)
    d = add(k1, d1) + add(k2[inner], q12[inner])
    vol = g["volume"]
    d = d + vol / dt
    b = b + vol / dt * f["rho_o"] * f["ui_o"] + f["source"] * vol - f["pi"] * vol
    b = b + d * (1.0 - urf) * phi / urf
    aval = torch.zeros(g["NONZ"], dtype=F64, device=DEV)
    aval[g["sid"][inner, 0]] = -q12[inner]
    aval[g["sid"][inner, 1]] = -q21[inner]
    aval[g["adia"]] = d[nb + 1:] / urf
    return {"aval": aval, "b": b[nb + 1:], "abou": torch.zeros(nb, dtype=F64, device=DEV),
            "asave": d[nb + 1:]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "calcps":
        return _exact_calcps(case, seed)
    if kind == "newuvw":
        return _exact_newuvw(case, seed)
    if kind == "batch":
        return {"xs": [_solution(p, val, b, "pressure" if m == "cg" else "transport")
                       for p, val, b, m, _ in _batch_systems(case, seed)], "status": None}
    if kind == "adjoint":
        gen = _rng(seed)
        p = _pattern(case["nx"], case["ny"], case["nz"])
        val, b = p.values(*_pressure(gen, case["nx"], case["ny"], case["nz"]))
        x = _solution(p, val, b, "pressure")
        lam = _solution(p, val, x - _uniform(gen, -1.0, 1.0, p.n), "pressure")
        row = torch.repeat_interleave(torch.arange(p.n, device=DEV), p.rowptr.diff().long())
        return {"x": x, "grad_val": -lam[row] * x[p.col.long()], "grad_b": lam}
    p, val, b = _system(case, seed)
    if case["maxiter"] <= 100:  # stopped early: the iterate of plain CG
        x = _cg(p.matrix(val), val[p.diag.long()], b, case["maxiter"], 0.0)
    else:
        x = _solution(p, val, b, case["system"])
    if kind == "legacy":  # x(-NB:N): the boundary part is not touched
        x = torch.nn.functional.pad(x, (_boundary_cells(case) + 1, 0)).cpu().numpy()
    return {"x": x, "niter": None, "status": None}
