"""Timed workloads of the library: fracture increments, smoother calls, batches and whole requests.

Every case is work a user's program hands to the library through `hpcrack_b200.solver`, `.serving`
or the C ABI (`hpcrack_b200.lib`).  The specimens are inclusion microstructures with the material
table, load schedule and multigrid parameters of `hpcrack_b200.microstructure`; sizes run from the
33^3 test specimens to the 257^3 benchmark specimen, cubes and uneven boxes.

Kinds:
  increments  a specimen at a saved state (checkpoint restore from pinned host memory) is taken
              through its next load increments and its fields are read back: the fracture loop
  smooth_u    one mechanical smoother call on the finest grid, grids copied in and out, as the
              function-level drop-in calls it
  smooth_d    the same for the phase field
  batch       several uneven specimens advanced together, one batched call per increment
  request     a whole served request: context, image to material, increments, fields, release

Fields read back: d and H, and u where the solve is FP64 throughout.  The supports (one x-fixed node
on the y = ya edge, one y-fixed node on the x = xb edge) leave a rigid rotation about the axis through
(xb, ya) free, and the precision form's FP32 cycle leaves rounding of its own size along it in u;
strains, and with them H, d and the reaction, do not see it.
"""
from __future__ import annotations

import numpy as np
import torch

from hpcrack_b200 import lib as _lib
from hpcrack_b200 import microstructure as ms
from hpcrack_b200 import serving
from hpcrack_b200.solver import (D, FD, FU, H, MECH_FAS, MECH_FCG, MECH_MIXED, R, RU, U, Batch, Hierarchy,
                                 precision_mg, step_params)

FORMS = {"fas": MECH_FAS, "fcg": MECH_FCG, "mixed": MECH_MIXED}
MG_U = (50, 4, 2, 1, 200)  # the reference configuration's cycles
MG_D = (10, 2, 1, 1, 200)
SMALL_K = 1e-6
LC = 2.0
VOXEL = 1e-6


def listed():
    return [
        # the smallest specimens users run (parameter studies, tests): launches and latency decide
        {"name": "inc33_fas", "kind": "increments", "nodes": "33x33x33", "form": "fas", "crack": 0, "steps": 1},
        # the 65^3 configuration in the reference's method and in the precision form
        {"name": "inc65_fas", "kind": "increments", "nodes": "65x65x65", "form": "fas", "crack": 0, "steps": 1},
        {"name": "inc65_mixed_x3", "kind": "increments", "nodes": "65x65x65", "form": "mixed", "crack": 0, "steps": 3},
        # an uneven box whose coarsest grid is too large for one thread block
        {"name": "inc257x129x65_fcg", "kind": "increments", "nodes": "257x129x65", "form": "fcg", "crack": 0,
         "steps": 1},
        # an odd coarsest grid (12 elements per axis), a size between the powers of two
        {"name": "inc97_mixed", "kind": "increments", "nodes": "97x97x97", "form": "mixed", "crack": 0, "steps": 1},
        {"name": "inc129_fas", "kind": "increments", "nodes": "129x129x129", "form": "fas", "crack": 0, "steps": 1},
        # the benchmark specimen (pre-crack, three phases: d starts non-zero) in the reference's method, and
        # its size in the precision form
        {"name": "crack257_fas", "kind": "increments", "nodes": "257x257x257", "form": "fas", "crack": 1, "steps": 1},
        {"name": "inc257_mixed", "kind": "increments", "nodes": "257x257x257", "form": "mixed", "crack": 0,
         "steps": 1},
        # function-level drop-in calls on one grid
        {"name": "smooth_u_161x97x65", "kind": "smooth_u", "nodes": "161x97x65", "iters": 4},
        {"name": "smooth_d_129", "kind": "smooth_d", "nodes": "129x129x129", "iters": 2},
        # a batch of uneven specimens, as the batched form runs them
        {"name": "batch6_mixed", "kind": "batch", "form": "mixed", "steps": 2,
         "sizes": "65x65x65,33x97x65,129x65x97,97x97x97,161x33x65,129x129x129"},
        # one served request from image to final fields
        {"name": "request65_mixed", "kind": "request", "nodes": "65x65x65", "form": "mixed", "steps": 4},
    ]


def _log_axis(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _draw_nodes(rng, lo=33, hi=2.2e6):
    """Box of lo^3 .. hi nodes: coarsest grids of 8 to 20 elements per axis, 2 to 4 levels above.  An even
    number of coarsest elements in x and y, so that the mid-edge supports are nodes of every level."""
    while True:
        target = _log_axis(rng, lo ** 3, hi)
        level = rng.randint(1, 4)
        n = [e * 2 ** level + 1 for e in (2 * rng.randint(4, 10), 2 * rng.randint(4, 10), rng.randint(8, 20))]
        if any(e % 2 for e in ms.hierarchy_for(n)[1][:2]):
            continue
        total = n[0] * n[1] * n[2]
        if 0.6 * target <= total <= min(1.5 * target, hi):
            return "%dx%dx%d" % tuple(n)


def draw(rng):
    kind = rng.choice(["increments"] * 4 + ["smooth_u", "smooth_d", "batch", "request"])
    if kind == "increments":
        form = rng.choice(["fas", "fcg", "mixed", "mixed"])
        return {"kind": kind, "nodes": _draw_nodes(rng), "form": form, "crack": int(form == "fas" and rng.random() < 0.3),
                "steps": 1 if form == "fas" else rng.randint(1, 3)}
    if kind in ("smooth_u", "smooth_d"):
        return {"kind": kind, "nodes": _draw_nodes(rng), "iters": rng.randint(1, 6)}
    if kind == "batch":
        sizes = ",".join(_draw_nodes(rng, hi=5e5) for _ in range(rng.randint(2, 6)))
        return {"kind": kind, "form": rng.choice(["fas", "mixed"]), "steps": 1, "sizes": sizes}
    return {"kind": kind, "nodes": _draw_nodes(rng, hi=5e5), "form": "mixed", "steps": rng.randint(2, 4)}


# ------------------------------------------------------------------------------------------ inputs
def _nodes(case, key="nodes"):
    return tuple(int(v) for v in case[key].split("x"))


def _image(nodes, seed, pores):
    """uint8 image (nz, ny, nx): one sphere per cell of a lattice, random radius and offset, so that no
    two overlap; radii 4 to 8 voxels at 65^3, scaled with the shortest axis; 5 to 24 % volume."""
    nx, ny, nz = nodes
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    rand = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    a = 16.0 * (min(nodes) - 1) / 64.0 + 1.0
    cells = [int(n / a) + 1 for n in (nz, ny, nx)]
    frac = 0.05 + 0.19 * float(rand(1))
    r = a * (0.25 + 0.25 * rand(*cells))
    r = torch.where(rand(*cells) < frac / 0.2455, r, torch.zeros_like(r))
    off = [(rand(*cells) - 0.5) * (a - 2 * r) for _ in range(3)]
    gray = torch.full(cells, ms.INCLUSION_GRAY, device="cuda", dtype=torch.uint8)
    if pores:
        gray[rand(*cells) < 0.2] = ms.PORE_GRAY
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in (nz, ny, nx)]
    ci = [(v / a).long() for v in ax]
    at = (ci[0][:, None, None], ci[1][None, :, None], ci[2][None, None, :])
    d2 = torch.zeros(nz, ny, nx, device="cuda", dtype=torch.float64)
    for q, shape in enumerate(((-1, 1, 1), (1, -1, 1), (1, 1, -1))):
        centre = (ci[q].double().view(shape) + 0.5) * a + off[q][at]
        d2 += (ax[q].view(shape) - centre) ** 2
    img = torch.where(d2 < r[at] ** 2, gray[at], torch.zeros_like(gray[at]))
    return img.cpu().numpy()


def _workload(nodes, seed, crack, steps, form="mixed"):
    level, enb = ms.hierarchy_for(nodes)
    # the driving energy passes its threshold Gc / (2 l) near 2.9 % strain in the plain matrix, earlier
    # beside inclusions: the first increment starts damage there, the next ones spread it; a pre-cracked
    # specimen damages at any load
    ut0, du = (1e-4, 1e-4) if crack else (0.021, 0.0002)
    ut0, du = ut0 * (nodes[2] - 1), du * (nodes[2] - 1)
    # the reference's method at the reference's own threshold |r|^2/|f|^2 <= 1e-6, the flexible forms
    # to |r|/|f| <= 1e-8 (FP64 cycle) and, so that d and H are settled to 1e-10 whatever the cycle's
    # rounding, 1e-11 (FP32 cycle)
    return ms.Workload("case", _image(nodes, seed, bool(crack)), enb, level, (0.0, 0.0, 0.0), VOXEL, LC, SMALL_K, MG_U,
                       MG_D, steps, ut0=ut0, du=du, mech_tol={"fas": 1e-6, "fcg": 1e-16, "mixed": 1e-22}[form], pf_tol=1e-16,
                       crack={"H": 1e6, "layer": (nodes[2] - 1) // 2, "xfrac": 0.5} if crack else None)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _host(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _read(h, field, buf):
    """hpc_download of every component of a finest field into a caller's pinned buffer."""
    lib = _lib.load()
    for comp in range(buf.shape[0] if buf.ndim == 2 else 1):
        row = buf[comp] if buf.ndim == 2 else buf
        _lib.check("hpc_download", lib.hpc_download(h.h, field, h.maxlevel, comp, row.ctypes.data_as(_lib._dp)))
    return buf


FIELDS = {"u": U, "d": D, "H": H}


def _outputs(n, form):
    """Pinned buffers of the fields a run of `form` reads back."""
    return {**({} if form == "mixed" else {"u": _host(3, n)}), "d": _host(n), "H": _host(n)}


def _fields(h, buffers):
    return {k: _read(h, FIELDS[k], b) for k, b in buffers.items()}


def _curve(outs):
    """Load, reaction and damage maxima of every increment (the F-U curve; the rest counts cycles)."""
    return np.array(outs)[..., :4]


def _mg_u(w, form):
    return w.mg_u if form == "fas" else precision_mg(w.maxlevel, w.element_nb, w.mg_u[4])


class _Specimen:
    """A context with its material, the pinned state it starts from and the buffers it is read into."""

    def __init__(self, nodes, seed, crack, steps, form):
        self.w = w = _workload(nodes, seed, crack, steps, form)
        self.h = Hierarchy(w.maxlevel, w.element_nb, x0=w.x_start)
        self.h.image_material(w.image, w.nodes, w.table(), w.voxel_size)
        n = self.h.n(w.maxlevel)
        zero = _pinned(np.zeros(n))
        self.start = {k: zero for k in Hierarchy.CHECKPOINT_FIELDS}
        if crack:
            Hc, dc = ms.precrack_fields(w)
            self.start.update(H=_pinned(Hc), d=_pinned(dc))
            self.start["d_old"] = self.start["d"]
        self.out = _outputs(n, form)
        self.mg = _mg_u(w, form)
        self.form = FORMS[form]

    def restore(self):
        self.h.checkpoint_restore(self.start, [0.0] * 6)

    def step(self, t):
        w = self.w
        return self.h.step(t, self.mg, w.mg_d, w.small_k, w.lc, w.voxel_size, ut0=w.ut0, dU=w.du, mech_tol=w.mech_tol,
                           pf_tol=w.pf_tol, mech_solver=self.form)

    def params(self, t):
        w = self.w
        return step_params(t, self.mg, w.mg_d, w.small_k, w.lc, w.voxel_size, ut0=w.ut0, dU=w.du, mech_tol=w.mech_tol,
                           pf_tol=w.pf_tol, mech_solver=self.form)

    def fields(self):
        return _fields(self.h, self.out)


def _smooth_fields(nodes, seed):
    """Displacement, phase field, regimes and history a smoother meets inside a run: a stretched bar with
    a local disturbance, damage in a band, zero damage far from it.  Arrays of (nz, ny, nx)."""
    nx, ny, nz = nodes
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 3)
    rand = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    z = torch.arange(nz, device="cuda", dtype=torch.float64).view(-1, 1, 1) / (nz - 1)
    y = torch.arange(ny, device="cuda", dtype=torch.float64).view(1, -1, 1) / (ny - 1)
    x = torch.arange(nx, device="cuda", dtype=torch.float64).view(1, 1, -1) / (nx - 1)
    one = torch.ones(nz, ny, nx, device="cuda", dtype=torch.float64)
    u = torch.stack([-0.2 * x * one, -0.2 * y * one, z * one]) + 1e-3 * (rand(3, nz, ny, nx) - 0.5)
    mid = 0.35 + 0.3 * float(rand(1))
    d = 0.9 * torch.exp(-(((z - mid) * (nz - 1)) / 4.0) ** 2) * (0.5 + 0.5 * rand(nz, ny, nx)) * one
    d = torch.where((z - mid).abs() * (nz - 1) > 16, torch.zeros_like(d), d)
    choice = torch.where(rand(nz, ny, nx) < 0.8, 0, torch.randint(1, 3, (nz, ny, nx), generator=gen, device="cuda"))
    hist = 20.0 * d * rand(nz, ny, nx)
    fd = 2.0 * hist
    for q, n in enumerate((nz, ny, nx)):  # element data: no value on the last planes
        hist.select(q, n - 1).zero_()
    return u, d, choice, hist, fd


def prepare(case, seed):
    kind = case["kind"]
    if kind == "increments":
        return {"case": case, "s": _Specimen(_nodes(case), seed, case["crack"], case["steps"], case["form"])}
    if kind == "batch":
        sizes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
        return {"case": case, "batch": Batch(),
                "s": [_Specimen(n, seed * 64 + i, 0, case["steps"], case["form"]) for i, n in enumerate(sizes)]}
    if kind == "request":
        w = _workload(_nodes(case), seed, 0, case["steps"])
        n = int(np.prod(w.nodes))
        return {"case": case, "w": w, "out": _outputs(n, case["form"])}
    nodes = _nodes(case)
    w = _workload(nodes, seed, 0, 1)
    h = Hierarchy(w.maxlevel, w.element_nb, x0=w.x_start)
    h.image_material(w.image, w.nodes, w.table(), w.voxel_size)
    u, d, choice, hist, fd = (v.cpu().numpy() for v in _smooth_fields(nodes, seed))
    n = h.n(w.maxlevel)
    st = {"case": case, "h": h, "d": _pinned(d.reshape(n))}
    if kind == "smooth_u":
        h.set(D, w.maxlevel, st["d"])
        h.set_choice(w.maxlevel, choice.reshape(n))
        st.update(u=_pinned(u.reshape(3, n)), f=_pinned(np.zeros((3, n))), u_out=_host(3, n), r_out=_host(3, n))
    else:
        h.set(H, w.maxlevel, hist.reshape(n))
        st.update(fd=_pinned(fd.reshape(n)), d_out=_host(n), r_out=_host(n))
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "increments":
        s = state["s"]
        s.restore()
        outs = [s.step(t) for t in range(case["steps"])]
        return {**s.fields(), "curve": _curve(outs)}
    if kind == "batch":
        for s in state["s"]:
            s.restore()
        outs = [state["batch"].step([s.h for s in state["s"]], [s.params(t) for s in state["s"]])
                for t in range(case["steps"])]
        return {"fields": [s.fields() for s in state["s"]], "curve": _curve(outs)}
    if kind == "request":
        w = state["w"]
        with Hierarchy(w.maxlevel, w.element_nb, x0=w.x_start) as h:
            outs = serving.run_request(h, w, case["steps"], mech_solver=FORMS[case["form"]])
            return {**_fields(h, state["out"]), "curve": _curve(outs)}
    h, L = state["h"], state["h"].maxlevel
    if kind == "smooth_u":
        h.set(U, L, state["u"])
        h.set(FU, L, state["f"])
        _, f_norm = h.pcg_u(L, SMALL_K, 1.0, case["iters"], 0, 0.0)
        return {"u": _read(h, U, state["u_out"]), "r": _read(h, RU, state["r_out"]), "f_norm": f_norm}
    h.set(D, L, state["d"])
    h.set(FD, L, state["fd"])
    _, fd_norm = h.pcg_d(L, LC, case["iters"], 1, 0.0)
    return {"d": _read(h, D, state["d_out"]), "r": _read(h, R, state["r_out"]), "fd_norm": fd_norm}


# ------------------------------------------------------------------------------------------- work
# Floating-point operations of one element: the mechanical action by sum factorisation (3 components
# forward and back, Hooke's law at 8 Gauss points), the phase-field action.
MECH_FLOPS, PF_FLOPS = 700.0, 250.0
# Cycles an increment takes to its tolerance, typical of the sizes above, by form.
CYCLES = {"fas": 4, "crack": 60, "fcg": 40, "mixed": 30}
# Bytes a smoother iteration cannot do without on one node, in values: moduli (nodal K, G, d), u, r, p,
# the inverse diagonal read and u, r, p written; times 8/7 for the coarser grids.
MECH_VALUES, PF_VALUES = 3 + 4 * 3 + 3 * 3, 2 + 4 + 3


def _increment_work(nodes, form, steps, crack=0):
    n = float(np.prod(nodes))
    nu = 6 if form == "fas" else 8
    applies = CYCLES["crack" if crack else form] * (nu + 2) * 8.0 / 7.0
    size = 4.0 if form == "mixed" else 8.0
    by = steps * (applies * n * MECH_VALUES * size + 5 * n * PF_VALUES * 8.0 + 14 * n * 8.0)
    return by, steps * (applies * n * MECH_FLOPS + 5 * n * PF_FLOPS)


def work(case):
    kind = case["kind"]
    if kind == "increments":
        by, fl = _increment_work(_nodes(case), case["form"], case["steps"], case["crack"])
        return {"bytes": by + 11 * 8.0 * float(np.prod(_nodes(case))), "flops": fl}
    if kind == "batch":
        total = [_increment_work(tuple(int(v) for v in s.split("x")), case["form"], case["steps"])
                 for s in case["sizes"].split(",")]
        return {"bytes": sum(t[0] for t in total), "flops": sum(t[1] for t in total)}
    if kind == "request":
        by, fl = _increment_work(_nodes(case), case["form"], case["steps"])
        return {"bytes": by, "flops": fl}
    n, it = float(np.prod(_nodes(case))), case["iters"] + 1
    if kind == "smooth_u":
        return {"bytes": it * n * MECH_VALUES * 8.0 + 12 * 8.0 * n, "flops": it * n * MECH_FLOPS}
    return {"bytes": it * n * PF_VALUES * 8.0 + 4 * 8.0 * n, "flops": it * n * PF_FLOPS}


# ------------------------------------------------------------------------------------------ exact
class _Grid:
    """Trilinear elements with 2x2x2 Gauss points on a unit-spaced grid, in plain FP64 torch."""

    def __init__(self, nodes):
        self.nodes = nx, ny, nz = nodes
        self.n = nx * ny * nz
        k, j, i = torch.meshgrid(torch.arange(nz - 1), torch.arange(ny - 1), torch.arange(nx - 1), indexing="ij")
        first = (i + j * nx + k * nx * ny).reshape(-1).cuda()
        self.first = first
        corners = [(a, b, c) for c in (0, 1) for b in (0, 1) for a in (0, 1)]
        self.conn = torch.stack([first + a + b * nx + c * nx * ny for a, b, c in corners])  # (8, E)
        t = [0.5 * (1 - 1 / np.sqrt(3.0)), 0.5 * (1 + 1 / np.sqrt(3.0))]
        N, dN = np.zeros((8, 8)), np.zeros((8, 8, 3))
        for g in range(8):
            p = (t[g & 1], t[(g >> 1) & 1], t[g >> 2])
            for m, abc in enumerate(corners):
                s = [p[q] if abc[q] else 1 - p[q] for q in range(3)]
                ds = [1.0 if abc[q] else -1.0 for q in range(3)]
                N[g, m] = s[0] * s[1] * s[2]
                dN[g, m] = ds[0] * s[1] * s[2], s[0] * ds[1] * s[2], s[0] * s[1] * ds[2]
        self.N, self.dN = torch.tensor(N).cuda(), torch.tensor(dN).cuda()

    def values(self, f):
        """Gauss-point values (8, E) of a nodal field, 0 at all 8 where a corner is exactly 0."""
        c = f.reshape(-1)[self.conn]
        return torch.where((c == 0).any(0), torch.zeros((), dtype=c.dtype, device=c.device), self.N @ c)

    def scatter(self, fe):
        out = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        for m in range(8):
            out.index_add_(0, self.conn[m], fe[m])
        return out

    def grads(self, u, g):
        """(3, 3, E): derivative q of component m at Gauss point g."""
        return torch.stack([self.dN[g].T @ u[m].reshape(-1)[self.conn] for m in range(3)])

    def mech(self, u, lam, mu):
        fe = torch.zeros(3, 8, self.conn.shape[1], dtype=torch.float64, device="cuda")
        for g in range(8):
            du = self.grads(u, g)
            tr = lam[g] * (du[0, 0] + du[1, 1] + du[2, 2])
            for m in range(3):
                s = torch.stack([mu[g] * (du[m, q] + du[q, m]) for q in range(3)])
                s[m] += tr
                fe[m] += 0.125 * (self.dN[g] @ s)
        return torch.stack([self.scatter(fe[m]) for m in range(3)])

    def mech_diag(self, lam, mu):
        fe = torch.zeros(3, 8, self.conn.shape[1], dtype=torch.float64, device="cuda")
        for g in range(8):
            sq = self.dN[g] ** 2
            for m in range(3):
                fe[m] += 0.125 * (torch.outer(sq[:, m], lam[g] + mu[g]) + torch.outer(sq.sum(1), mu[g]))
        return torch.stack([self.scatter(fe[m]) for m in range(3)])

    def field(self, x, aw, bw):
        c = x.reshape(-1)[self.conn]
        fe = torch.zeros_like(c)
        for g in range(8):
            fe += torch.outer(self.N[g], aw[g] * (self.N[g] @ c)) + self.dN[g] @ (bw[g] * (self.dN[g].T @ c))
        return self.scatter(fe)

    def field_diag(self, aw, bw):
        fe = sum(torch.outer(self.N[g] ** 2, aw[g]) + torch.outer((self.dN[g] ** 2).sum(1), bw[g]) for g in range(8))
        return self.scatter(fe)

    def fixed(self):
        """(3, n) mask of the Dirichlet rows, and the mask of the top plane's u_z."""
        nx, ny, nz = self.nodes
        m = torch.zeros(3, nz, ny, nx, dtype=torch.bool, device="cuda")
        if nx % 2:
            m[0, 0, 0, (nx - 1) // 2] = True
        if ny % 2:
            m[1, 0, (ny - 1) // 2, nx - 1] = True
        m[2, 0] = m[2, nz - 1] = True
        top = torch.zeros(3, nz, ny, nx, dtype=torch.bool, device="cuda")
        top[2, nz - 1] = True
        return m.view(3, -1), top.view(3, -1)


def _nodal_material(image):
    """Nodal K, G, Gc of the labels, E scaled by the voxel size."""
    lab = torch.from_numpy(image).cuda().reshape(-1)
    out = [torch.zeros(lab.numel(), dtype=torch.float64, device="cuda") for _ in range(3)]
    for gray, m in ((ms.MATRIX_GRAY, ms.MATRIX), (ms.PORE_GRAY, ms.PORE), (ms.INCLUSION_GRAY, ms.INCLUSION)):
        at = lab == gray
        out[0][at] = m.E * VOXEL / (3 * (1 - 2 * m.nu))
        out[1][at] = m.E * VOXEL / (2 * (1 + m.nu))
        out[2][at] = m.gc
    return out


def _degraded(grid, K, G, d, choice):
    """(lam, mu) at the Gauss points: K and G degraded by g(d) by regime (0 both, 1 shear, 2 none)."""
    Kg, Gg = grid.values(K), grid.values(G)
    gd = (1 - SMALL_K) * (1 - grid.values(d).clamp(0, 1)) ** 2 + SMALL_K
    ch = choice.reshape(-1)[grid.first]
    Kd, Gd = torch.where(ch == 0, gd * Kg, Kg), torch.where(ch == 2, Gg, gd * Gg)
    return Kd - 2.0 / 3.0 * Gd, Gd


def _pcg(apply, x, r, inv, iters, zero=None, tol=0.0):
    rz = (r * inv * r).sum()
    p = torch.zeros_like(r)
    beta = 0.0
    start = (r * r).sum()
    for _ in range(iters):
        p = r * inv + beta * p
        w = apply(p)
        alpha = rz / (p * w).sum()
        x = x + alpha * p
        r = r - alpha * w
        if zero is not None:
            r[zero] = 0.0
        rz_new = (r * inv * r).sum()
        beta, rz = rz_new / rz, rz_new
        if tol and (r * r).sum() <= tol * start:
            break
    return x, r


def exact(case, seed):
    """Smoother calls of any size, and first increments of uncracked specimens small enough to solve by
    plain conjugate gradients; None elsewhere."""
    kind = case["kind"]
    if kind in ("batch", "request"):
        return None
    nodes = _nodes(case)
    n = int(np.prod(nodes))
    if kind == "increments" and (case["crack"] or case["steps"] != 1 or n > 300000):
        return None
    w = _workload(nodes, seed, 0, 1, case.get("form", "fas"))
    grid = _Grid(nodes)
    K, G, gc = _nodal_material(w.image)
    fix, top = grid.fixed()
    if kind == "smooth_u":
        u, d, choice, _, _ = _smooth_fields(nodes, seed)
        lam, mu = _degraded(grid, K, G, d.reshape(-1), choice)
        inv = 1.0 / grid.mech_diag(lam, mu)
        u = u.reshape(3, -1).clone()
        u[fix] = 0.0
        u[top] = 1.0
        Ku = grid.mech(u, lam, mu)
        f = torch.where(fix, Ku, torch.zeros_like(Ku))
        u, r = _pcg(lambda p: grid.mech(p, lam, mu), u, f - Ku, inv, case["iters"], zero=fix)
        return {"u": u, "r": r, "f_norm": float((f * f).sum())}
    gcg = grid.values(gc)
    if kind == "smooth_d":
        _, d, _, hist, fd = _smooth_fields(nodes, seed)
        aw = 0.125 * (2 * hist.reshape(-1)[grid.first] + gcg / LC)
        bw = 0.125 * gcg * LC
        d, fd = d.reshape(-1), fd.reshape(-1)
        inv = 1.0 / grid.field_diag(aw, bw)
        d, r = _pcg(lambda p: grid.field(p, aw, bw), d, fd - grid.field(d, aw, bw), inv, case["iters"])
        return {"d": d, "r": r, "fd_norm": float((fd * fd).sum())}
    # the first increment: u at unit top displacement, history at the load, d
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    lam, mu = _degraded(grid, K, G, zero, zero.long())
    u = torch.zeros(3, n, dtype=torch.float64, device="cuda")
    u[top] = 1.0
    r = -grid.mech(u, lam, mu)
    r[fix] = 0.0
    inv = 1.0 / grid.mech_diag(lam, mu)
    u, _ = _pcg(lambda p: grid.mech(p, lam, mu), u, r, inv, 3000, zero=fix, tol=1e-26)
    Kg, Gg = grid.values(K), grid.values(G)
    mean = torch.zeros(grid.conn.shape[1], dtype=torch.float64, device="cuda")
    for g in range(8):
        du = w.ut0 * grid.grads(u, g)
        e = 0.5 * (du + du.transpose(0, 1))
        tr = e[0, 0] + e[1, 1] + e[2, 2]
        dev2 = (e * e).sum((0, 1)) - tr * tr / 3
        mean += 0.125 * (0.5 * Kg[g] * tr.clamp(min=0) ** 2 + Gg[g] * dev2 - 0.5 * gcg[g] / LC)
    hist = mean.clamp(min=0)
    fd = grid.scatter(0.125 * 2 * hist * grid.N.sum(0)[:, None])
    aw, bw = 0.125 * (2 * hist + gcg / LC), 0.125 * gcg * LC
    d, _ = _pcg(lambda p: grid.field(p, aw, bw), zero, fd, 1.0 / grid.field_diag(aw, bw), 500, tol=1e-28)
    H_nodes = zero.clone()
    H_nodes[grid.first] = hist
    return {**({} if case["form"] == "mixed" else {"u": u}), "d": d, "H": H_nodes, "curve": None}
