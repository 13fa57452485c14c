"""Performance cases: whole time steps of flow cases through ``higflow_b200.engine``.

Every case is one pass of the engine's main use: a state goes in (velocity,
pressure, pressure increment, conformation kernel; a restart file or the host
solver's fields), a number of time steps run on the GPU, and the fields come
back at the output point.  The programs are lid-driven boxes on uniform grids,
built here in the recorded form (one stencil row per query, its weights unique
to its last bits, order-2 least-squares rows of up to 45 points in 2D and 110
in 3D, wall values in the rows' boundary terms), so that no recording host is
needed.  A program's engine case (the handle) is kept as a user's program keeps
it; each pass writes the whole state first, so a pass depends on its inputs only.
"""
import functools
import math

import numpy as np
import torch

from higflow_b200 import engine
from higflow_b200 import program as hp


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _case(name, flow, sides, steps, precision="plain", scheme="explicit", per_step=False, limits=""):
    return dict(name=name, flow=flow, sides=sides, steps=steps, precision=precision, scheme=scheme,
                per_step=per_step, limits=limits)


def listed():
    return [
        # the link-time replacement of a HigFlow main's time loop on a small
        # 2D case: the time step is set and the solver's result read each step
        _case("drop_in_33", "newtonian", "33x33", 4, per_step=True),
        # one 2D Newtonian cavity at the suite's standard size
        _case("newtonian_64", "newtonian", "64x64", 20),
        # the largest 2D case of the served stream
        _case("newtonian_512_mixed", "newtonian", "512x512", 5, "mixed"),
        # the batched population (Giesekus, side log-uniform in [32, 256]) at
        # its side quantiles, in both forms
        _case("giesekus_batch_mixed", "giesekus", "55,45,114,122,183,77,48,63,140,224,82,107,209,131,171,"
              "67,94,51,34,239,100,196,32,160,37,42,256,72,150,39,59,88", 6, "mixed"),
        _case("giesekus_batch_plain", "giesekus", "47,219,77,61,155,129,33,101", 6),
        # one mid-size viscoelastic case in the plain form (a production run
        # that is checked against the CPU solver)
        _case("oldroyd_129", "oldroyd", "129x129", 10),
        # the channel's shape: 4:1 box, square cells
        _case("oldroyd_260x65_mixed", "oldroyd", "260x65", 10, "mixed"),
        # 3D cavity at the suite's 3D size, and a 3D viscoelastic one
        _case("newtonian_32cube_mixed", "newtonian", "32x32x32", 4, "mixed"),
        _case("oldroyd_17cube", "oldroyd", "17x17x17", 3),
        # creeping flow beyond the explicit bound: semi-implicit velocity
        _case("semi_implicit_96", "oldroyd", "96x96", 4, scheme="semi_implicit"),
        # a served cohort: requests of several sizes and step counts in one batch
        _case("cohort_limits_mixed", "newtonian", "64,91,128,181,256", 8, "mixed", limits="3,8,5,8,2"),
    ]


def draw(rng):
    """One more case: single 2D boxes of side 32 to 512, batches, cohorts under
    step limits, 3D boxes, both forms."""
    logint = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["single", "single", "box", "batch", "cohort", "cube", "implicit"])
    precision = rng.choice(["plain", "mixed"])
    flow = rng.choice(["newtonian", "oldroyd", "giesekus"])
    steps = rng.randint(3, 12)
    scheme, limits = "explicit", ""
    if kind == "single":
        n = logint(32, 400 if flow == "newtonian" else 256)
        sides, steps = f"{n}x{n}", max(2, min(steps, 300000 // (n * n)))
    elif kind == "box":
        n = logint(24, 90)
        sides = f"{4 * n + rng.randint(0, 3)}x{n}"
    elif kind == "cube":
        n = rng.randint(12, 28) if flow == "newtonian" else rng.randint(9, 16)
        sides, steps = f"{n}x{n}x{n}", min(steps, 4)
    elif kind == "implicit":
        n = logint(32, 128)
        sides, steps, scheme, precision = f"{n}x{n}", min(steps, 4), "semi_implicit", "plain"
    else:
        count = rng.randint(3, 9)
        sides = ",".join(str(logint(32, 180)) for _ in range(count))
        steps = min(steps, 8)
        if kind == "cohort":
            limits = ",".join(str(rng.randint(1, steps)) for _ in range(count))
    return dict(flow=flow, sides=sides, steps=steps, precision=precision, scheme=scheme, per_step=False, limits=limits)


def _shapes(case):
    out = []
    for s in case["sides"].split(","):
        v = [int(x) for x in s.split("x")]
        out.append(tuple(v * 2 if len(v) == 1 else v))
    return out


def _physics(case, shape, i):
    """Parameters of instance i (fixed by the case: the inputs are the fields)."""
    D, h = len(shape), 1.0 / max(shape)
    ve = case["flow"] != "newtonian"
    implicit = case["scheme"] == "semi_implicit"
    Re = 0.01 if implicit else 1.0 if ve else 100.0
    dt = 0.2 * h * h if implicit else 0.2 * min(Re * h * h / 4.0, h)
    par = {k: hp._PARAM_DEFAULTS.get(k, 0.0) for k in hp._PARAM_NAMES}
    par.update(dim=D, flowtype=hp.VISCOELASTIC if ve else hp.NEWTONIAN, projtype=hp.INCREMENTAL,
               convecdiscrtype=hp.SECOND_ORDER, secondconvecdiscrtype=hp.CUBISTA,
               ve_model=hp.GIESEKUS if case["flow"] == "giesekus" else hp.OLDROYD_B,
               ve_convecdiscrtype=hp.CELL_CUBISTA, kernel=hp.KERNEL_LOG if ve else 0, Re=Re, dt=dt,
               De=0.3 + 0.13 * (i % 12), beta=0.1 if case["flow"] == "giesekus" else 1.0 / 9.0, kernel_tol=1e-2,
               alpha=0.05 + 0.035 * (i % 12), epsilon=0.25, xi=0.0,
               tempdiscrtype=hp.SEMI_IMPLICIT_EULER if implicit else hp.EXPLICIT_EULER)
    return par, h


# ---------------------------------------------------------------------------
# step programs of lid-driven boxes on uniform grids
# ---------------------------------------------------------------------------
_LID = 1.0      # u[0] on the upper face of the last axis


def _wls(off, lo, hi, D):
    """Least-squares rows at a query ``off`` (lattice units from its anchor
    point), one per class: (relative point indices, weights).  lo / hi:
    lattice points on either side of the anchor, per class and axis."""
    m, R = (45, 7) if D == 2 else (110, 5)
    box = np.stack([g.ravel() for g in np.meshgrid(*[np.arange(-R, R + 1)] * D, indexing="ij")], 1)
    d2 = ((box - np.asarray(off)) ** 2).sum(1)
    order = np.lexsort(tuple(box.T) + (np.round(d2, 9),))
    box, d2 = box[order], d2[order]
    ok = np.ones((len(lo), len(box)), bool)
    for k in range(D):
        ok &= (box[None, :, k] >= -lo[:, None, k]) & (box[None, :, k] <= hi[:, None, k])
    pick = np.argsort(~ok, axis=1, kind="stable")[:, :m]
    good = np.take_along_axis(ok, pick, 1)
    x = box[pick] - np.asarray(off)
    basis = [np.ones(x.shape[:2])] + [x[..., k] for k in range(D)]
    basis += [x[..., a] * x[..., b] for a in range(D) for b in range(a, D)]
    B = np.stack(basis, -1)
    w = np.where(good, 1.0 / np.maximum(d2[pick], 0.25) ** 2, 0.0)
    N = np.einsum("cmi,cm,cmj->cij", B, w, B)
    e0 = np.zeros(B.shape[-1])
    e0[0] = 1.0
    c = np.linalg.solve(N, np.broadcast_to(e0, (len(lo), len(e0)))[..., None])[..., 0]
    return box[pick], np.einsum("cmi,ci->cm", B, c) * w, good


class _Rows:
    """The program's general rows, one template per row."""

    def __init__(self, rng):
        self.rng, self.n, self.rhs, self.len, self.col, self.w = rng, 0, [], [], [], []
        self._const = {}

    def add(self, cols, w, keep, rhs):
        k = len(cols)
        self.rhs.append(np.broadcast_to(np.asarray(rhs, float), (k,)))
        self.len.append(keep.sum(1))
        self.col.append(cols[keep].astype(np.int32))
        # a recorded row is fitted at its own coordinates: its weights are its
        # own in the last bits
        ulp = 1.0 + 2.2e-16 * self.rng.integers(-3, 4, size=w.shape)
        self.w.append((w * ulp)[keep])
        self.n += k
        return -(np.arange(self.n - k, self.n) + 1)

    def const(self, value):
        """Code of the row without entries whose value is ``value``."""
        if value not in self._const:
            self._const[value] = int(self.add(np.zeros((1, 1), int), np.zeros((1, 1)), np.zeros((1, 1), bool), -value)[0])
        return self._const[value]

    def unit(self, cols, w, value):
        """Rows of one entry: w f[col] + value."""
        k = len(cols)
        return self.add(cols.reshape(-1, 1), np.full((k, 1), float(w)), np.ones((k, 1), bool), -value)

    def lattice(self, idx, off, dims, wall):
        """Least-squares rows on a field lattice of ``dims`` points (axis
        ``wall``: known zero values one step outside either end), anchored at
        the points ``idx`` (rows x D)."""
        D = len(dims)
        far = 8 if D == 2 else 6
        ext = np.array([1 if k == wall else 0 for k in range(D)])
        lo = np.minimum(idx + ext, far)
        hi = np.minimum(np.asarray(dims) - 1 - idx + ext, far)
        key, inv = np.unique(np.concatenate([lo, hi], 1), axis=0, return_inverse=True)
        inv = inv.reshape(-1)
        rel, w, good = _wls(off, key[:, :D], key[:, D:], D)
        p = idx[:, None, :] + rel[inv]
        keep = good[inv] & ((p >= 0) & (p < np.asarray(dims))).all(-1)
        strides = np.array([int(np.prod(dims[k + 1:])) for k in range(D)])
        return self.add((np.where(keep[..., None], p, 0) * strides).sum(-1), w[inv], keep, 0.0)


@functools.lru_cache(maxsize=40)
def _program(flow, scheme, shape, index):
    """One box's step program (hp.Program), cells and facets in row-major order."""
    par, h = _physics(dict(flow=flow, scheme=scheme), shape, index)
    D, ve, n = len(shape), flow != "newtonian", shape
    rows = _Rows(np.random.default_rng(7))
    fdims = [tuple(n[k] - (k == d) for k in range(D)) for d in range(D)]
    grid = lambda dims: np.stack([g.ravel() for g in np.meshgrid(*[np.arange(m) for m in dims], indexing="ij")], 1)  # noqa: E731
    flat = lambda idx, dims: np.ravel_multi_index(tuple(idx.T), dims)  # noqa: E731
    zero = rows.const(0.0)

    def shift(idx, *moves):
        idx = idx.copy()
        for k, s in moves:
            idx[:, k] += s
        return idx

    def facet(g, idx):
        """Codes of u[g] at lattice points idx of its facets, walls and one or
        two points beyond them included (linear through the wall value)."""
        dims = fdims[g]
        out = np.empty(len(idx), np.int64)
        inside = ((idx >= 0) & (idx < np.asarray(dims))).all(1)
        out[inside] = flat(idx[inside], dims)
        out[~inside] = zero
        onwall = (idx[:, g] == -1) | (idx[:, g] == dims[g])
        for k in range(D):
            for side in (0, 1):
                t = -idx[:, k] if side == 0 else idx[:, k] - dims[k] + 1      # points outside
                lid = _LID if (g == 0 and k == D - 1 and side == 1) else 0.0
                others = np.ones(len(idx), bool)
                for q in range(D):
                    if q != k:
                        others &= (idx[:, q] >= 0) & (idx[:, q] < dims[q])
                for steps in (1, 2):
                    sel = others & (t == steps) & ~onwall
                    if not sel.any():
                        continue
                    near = idx[sel].copy()
                    near[:, k] = 0 if side == 0 else dims[k] - 1
                    ratio = steps - 1.0 if k == g else 2.0 * steps - 1.0
                    out[sel] = rows.unit(flat(near, dims), -ratio, (1.0 + ratio) * lid)
        return out

    beyond = {}

    def outside_cells(k, side, steps):
        """Codes of a cell field ``steps`` cells outside a wall, by wall cell."""
        if (k, side, steps) not in beyond:
            dims = tuple(1 if q == k else n[q] for q in range(D))
            idx = grid(dims)
            idx[:, k] = 0 if side == 0 else n[k] - 1
            off = [0.0] * D
            off[k] = float(-steps if side == 0 else steps)
            beyond[k, side, steps] = rows.lattice(idx, off, n, -1).reshape(dims)
        return beyond[k, side, steps]

    def cell(idx):
        """Codes of a cell field at cell indices, up to two cells outside one wall."""
        out = np.full(len(idx), zero, np.int64)
        inside = ((idx >= 0) & (idx < np.asarray(n))).all(1)
        out[inside] = flat(idx[inside], n)
        for k in range(D):
            for side in (0, 1):
                t = -idx[:, k] if side == 0 else idx[:, k] - n[k] + 1
                for steps in (1, 2):
                    sel = ~inside & (t == steps)
                    if sel.any():
                        at = [idx[sel, q] if q != k else np.zeros(sel.sum(), int) for q in range(D)]
                        out[sel] = outside_cells(k, side, steps)[tuple(at)]
        return out

    # u[d] at the cell centres: anchored at the facet below (the wall for the first)
    centre = []
    for d in range(D):
        idx = grid(n)
        idx[:, d] -= 1
        off = [0.0] * D
        off[d] = 0.5
        centre.append(rows.lattice(idx, off, fdims[d], d).reshape(n))
    # u[g] at the edge points between the facets normal to g and to d
    corner = {}
    for d in range(D):
        for g in range(D):
            if g != d:
                dims = tuple(n[k] - (k in (g, d)) for k in range(D))
                off = [0.0] * D
                off[d] = 0.5
                corner[d, g] = rows.lattice(grid(dims), off, fdims[g], g).reshape(dims)

    vel, vflags, vdelta = [], [], []
    for d in range(D):
        I = grid(fdims[d])
        nf, own = len(I), flat(I, fdims[d])
        S = np.zeros((hp.v_nslot(D, ve), nf), np.int64)
        left, right = flat(I, n), flat(shift(I, (d, 1)), n)
        S[hp.V_FU], S[hp.V_PL], S[hp.V_PR], S[hp.V_FL], S[hp.V_FR] = own, left, right, left, right
        flags = np.zeros(nf, np.uint32)
        for g in range(D):
            b = hp.V_BLK0 + hp.V_NB * g
            if g != d:
                for q, (sd, sg) in enumerate(((1, 0), (1, -1), (0, 0), (0, -1))):
                    S[b + hp.V_V4 + q] = facet(g, shift(I, (d, sd), (g, sg)))
            for q, (slot, s) in enumerate(((hp.V_UL, -1), (hp.V_UR, 1), (hp.V_ULL, -2), (hp.V_URR, 2))):
                J = shift(I, (g, s))
                S[b + slot] = facet(d, J)
                wall = 1 if g == d else 0
                inf = (J[:, g] >= -wall) & (J[:, g] < fdims[d][g] + wall)
                flags |= (inf.astype(np.uint32) << np.uint32(4 * g + q))
            for slot, s in ((hp.V_VCR, 1), (hp.V_VCL, 0)):
                if g == d:
                    S[b + slot] = centre[d][tuple(shift(I, (d, s)).T)]
                else:
                    J = shift(I, (g, s - 1))
                    ok = (J[:, g] >= 0) & (J[:, g] < n[g] - 1)
                    S[b + slot] = zero
                    S[b + slot][ok] = corner[d, g][tuple(J[ok].T)]
            if ve:
                b = hp.v_nslot(D, False) + hp.V_NS * g
                if g == d:
                    S[b:b + 2], S[b + 2:b + 4] = left, right
                else:
                    for q, (sd, sg) in enumerate(((0, -1), (1, -1), (0, 1), (1, 1))):
                        S[b + q] = cell(shift(I, (d, sd), (g, sg)))
        vel.append(S.astype(np.int32))
        vflags.append(flags)
        vdelta.append(np.zeros(nf, np.uint16))

    I = grid(n)
    nc = len(I)
    div = np.zeros((2 * D, nc), np.int64)
    for d in range(D):
        div[2 * d], div[2 * d + 1] = facet(d, shift(I, (d, -1))), facet(d, I)
    cells = cflags = None
    if ve:
        C = np.zeros((hp.c_nslot(D), nc), np.int64)
        C[hp.C_SELF] = np.arange(nc)
        cflags = np.zeros(nc, np.uint32)
        pair = 0
        for d in range(D):
            b = hp.C_BLK0 + hp.C_NB * d
            C[b + hp.C_UVL], C[b + hp.C_UVR] = div[2 * d], div[2 * d + 1]
            for q, (slot, s) in enumerate(((hp.C_KL, -1), (hp.C_KR, 1), (hp.C_KLL, -2), (hp.C_KRR, 2))):
                J = shift(I, (d, s))
                C[b + slot] = cell(J)
                cflags |= ((J[:, d] >= 0) & (J[:, d] < n[d])).astype(np.uint32) << np.uint32(4 * d + q)
            for g in range(D):
                if g != d:
                    b2 = hp.C_BLK0 + hp.C_NB * D + hp.C_NQ * pair
                    pair += 1
                    for q, (sd, sg) in enumerate(((0, -1), (-1, -1), (0, 1), (-1, 1))):
                        C[b2 + q] = facet(d, shift(I, (d, sd), (g, sg)))
        cells = C.astype(np.int32)

    # Poisson rows: Neumann walls, one cell pinned
    pin = int(np.ravel_multi_index(tuple((m - 1) // 2 for m in n), n))
    cols = [np.arange(nc)]
    keep = [np.ones(nc, bool)]
    for d in range(D):
        for s in (1, -1):
            J = shift(I, (d, s))
            ok = (J[:, d] >= 0) & (J[:, d] < n[d])
            cols.append(flat(np.where(ok[:, None], J, 0), n))
            keep.append(ok)
    cols, keep = np.stack(cols, 1), np.stack(keep, 1)
    vals = np.where(keep, 1.0 / (h * h), 0.0)
    vals[:, 0] = -(keep.sum(1) - 1) / (h * h)
    keep[pin] = False
    ptr = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int64)
    return hp.Program(
        par=par, ncell=nc, nfacet=[int(np.prod(f)) for f in fdims] + [0] * (3 - D),
        delta=np.full((1, D), h), row_tmpl=np.arange(rows.n, dtype=np.int32), row_base=np.zeros(rows.n, np.int32),
        row_rhs=np.concatenate(rows.rhs), tmpl_ptr=np.concatenate([[0], np.cumsum(np.concatenate(rows.len))]).astype(np.int64),
        tmpl_col=np.concatenate(rows.col), tmpl_w=np.concatenate(rows.w), vel_slots=vel, vel_flags=vflags,
        vel_delta=vdelta, div_slots=div.astype(np.int32), cell_delta=np.zeros(nc, np.uint16), p_ptr=ptr,
        p_col=cols[keep].astype(np.int32), p_val=vals[keep], p_brhs=np.zeros(nc), pin_row=pin, pin_value=0.0,
        cell_slots=cells, cell_flags=cflags)


def _programs(case):
    return [_program(case["flow"], case["scheme"], s, i) for i, s in enumerate(_shapes(case))]


# ---------------------------------------------------------------------------
# inputs: a developed state (smooth divergence-free velocity at rest on the
# walls, smooth pressure, conformation with distinct principal stretches)
# ---------------------------------------------------------------------------
def _modes(rng, shape, pos, kind, terms=4):
    """A smooth random field on the tensor grid of positions ``pos`` (per axis, in [0, 1])."""
    f = np.zeros([len(p) for p in pos])
    for _ in range(terms):
        t = rng.uniform(-1.0, 1.0)
        for k, p in enumerate(pos):
            m = int(rng.integers(1, 4))
            v = np.sin(np.pi * p) * np.sin(m * np.pi * p) if kind == "wall" else np.cos(m * np.pi * p + rng.uniform(0, 1))
            t = t * v.reshape([-1 if q == k else 1 for q in range(len(pos))])
        f = f + t
    return f / terms


def _state(prog, shape, rng):
    D = len(shape)
    c = [(np.arange(m) + 0.5) / m for m in shape]
    nodes = [np.arange(m + 1) / m for m in shape[:2]] + c[2:]
    psi = _modes(rng, shape, nodes, "wall") * 0.3
    fields = {}
    u = [np.diff(psi, axis=1)[1:-1] * shape[1], -np.diff(psi, axis=0)[:, 1:-1] * shape[0]]
    if D == 3:
        u.append(np.zeros((shape[0], shape[1], shape[2] - 1)))
    for d in range(D):
        fields[hp.FIELD_U, d] = u[d].ravel()
    fields[hp.FIELD_P, 0] = _modes(rng, shape, c, "free").ravel()
    fields[hp.FIELD_DP, 0] = np.zeros(prog.ncell)
    if prog.viscoelastic:
        for i in range(D):
            for j in range(i, D):
                k = 0.15 * _modes(rng, shape, c, "free").ravel()
                if i == j:
                    k += 0.8 - 0.7 * i
                fields[hp.FIELD_KERNEL, i * D + j] = k
                fields[hp.FIELD_KERNEL, j * D + i] = k
    return fields


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    parts = [_state(p, s, rng) for p, s in zip(_programs(case), _shapes(case))]
    return parts, {k: np.concatenate([q[k] for q in parts]) for k in parts[0]}


@functools.lru_cache(maxsize=2)
def _handle(key):
    case = dict(key)
    progs = _programs(case)
    prog = progs[0] if len(progs) == 1 else hp.Program.concatenate(progs)
    prec = hp.PREC_MIXED if case["precision"] == "mixed" else hp.PREC_FP64
    return engine.Case(prog, engine.options(precision=prec))


def prepare(case, seed):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    limits = [int(x) for x in case["limits"].split(",")] if case["limits"] else None
    return dict(case=_handle(key), fields=_inputs(case, seed)[1], steps=case["steps"], per_step=case["per_step"],
                limits=limits)


def run(state):
    c = state["case"]
    for (fid, comp), v in state["fields"].items():
        c.set(fid, comp, v)
    if state["limits"]:
        c.set_step_limits(state["limits"])
    if state["per_step"]:
        dt = c.prog.par["dt"]
        for _ in range(state["steps"]):
            c.set_timestep(dt)
            c.step(1)
            c.instance_result(0)
    else:
        c.step(state["steps"])
    D = c.prog.dim
    out = {f"u{d}": c.get(hp.FIELD_U, d) for d in range(D)}
    out["p"] = c.get(hp.FIELD_P, 0)
    if c.prog.viscoelastic:
        for i in range(D):
            for j in range(i, D):
                out[f"K{i}{j}"] = c.get(hp.FIELD_KERNEL, i * D + j)
    return out


def work(case):
    """Per step: every general row's entries (column and weight), every slot
    code, the state read and written once, u* and the Poisson unknown written
    and read once; the state's transfer in and out."""
    w = 8 if case["precision"] == "plain" else 4
    b = f = 0.0
    limits = [int(x) for x in case["limits"].split(",")] if case["limits"] else None
    for i, p in enumerate(_programs(case)):
        D, nf = p.dim, sum(p.nfacet)
        comps = D * (D + 1) // 2 if p.viscoelastic else 0
        entries = len(p.tmpl_col)
        step = entries * (4 + w) + 4 * sum(s.size for s in p.vel_slots) + 4 * p.div_slots.size + 8 * 4 * nf
        step += 8 * p.ncell * (4 + (4 * comps if comps else 0)) + 4 * (p.cell_slots.size if comps else 0)
        flops = 2 * entries + 40 * D * nf + p.ncell * (20 * D + (200 * D * D if comps else 0))
        k = limits[i] if limits else case["steps"]
        b += k * step + 8 * (2 * nf + p.ncell * (3 + 2 * comps))
        f += k * flops
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same steps in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _eigh(a):
    """Eigenvalues and vectors of a batch of symmetric matrices, some at a time."""
    parts = [torch.linalg.eigh(x) for x in a.split(8192)]
    return torch.cat([q[0] for q in parts]), torch.cat([q[1] for q in parts])


class _Exact:
    """One box: the reference's step, formula by formula, over the program's
    rows; the Poisson and velocity systems solved in their 1D eigenvectors."""

    def __init__(self, prog, shape, dev):
        self.p, self.shape, self.dev, self.D = prog, shape, dev, prog.dim
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.ptr, self.col, self.w, self.rhs = (self.t(a) for a in (prog.tmpl_ptr, prog.tmpl_col.astype(np.int64),
                                                                    prog.tmpl_w, prog.row_rhs))
        self.h, self.par = float(prog.delta[0, 0]), prog.par
        self.vs = [self.t(s.astype(np.int64)) for s in prog.vel_slots]
        self.ds = self.t(prog.div_slots.astype(np.int64))
        self.vf = [self.t(f.astype(np.int64)) for f in prog.vel_flags]
        if prog.viscoelastic:
            self.cs, self.cf = self.t(prog.cell_slots.astype(np.int64)), self.t(prog.cell_flags.astype(np.int64))

    def q(self, code, f):
        out = f[code.clamp(min=0)]
        g = (code < 0).nonzero()[:, 0]
        if len(g):
            r = -code[g] - 1
            a, m = self.ptr[r], self.ptr[r + 1] - self.ptr[r]
            k = torch.arange(int(m.max()) if len(m) else 0, device=self.dev)
            at = (a[:, None] + k).clamp(max=max(len(self.col) - 1, 0))
            v = torch.where(k < m[:, None], f[self.col[at]] * self.w[at], 0.0).sum(1)
            out = out.index_put((g,), v - self.rhs[r])
        return out

    @staticmethod
    def eq(a, b):
        return (a - b).abs() < 1e-12

    def cubista(self, up, c, dn, flux, far=True, near=True):
        """Flux times the CUBISTA face value between c (upwind cell) and dn,
        up behind c; ``far`` / ``near``: see the callers' domain tests."""
        fi = torch.where(self.eq(dn, up), -1.0, (c - up) / (dn - up))
        low = torch.where(far, 1.75 * c - 0.75 * up, c)
        mid = torch.where(far & near, 0.75 * c + 0.375 * dn - 0.125 * up, c)
        high = torch.where(near, 0.25 * c + 0.75 * dn, c)
        v = torch.where(fi < 0.375, low, torch.where(fi <= 0.75, mid, high))
        return flux * torch.where((fi <= 0) | (fi >= 1), c, v)

    def velocity(self, u, p, S):
        D, h, par, out = self.D, self.h, self.par, []
        true = torch.ones((), dtype=torch.bool, device=self.dev)
        for d in range(D):
            s, fl, c = self.vs[d], self.vf[d], u[d]
            first = torch.zeros_like(c, dtype=torch.bool)
            dp = (self.q(s[hp.V_PR], p) - self.q(s[hp.V_PL], p)) / h
            cub, upw, diff, tens, stopped = 0.0, 0.0, 0.0, 0.0, first
            for g in range(D):
                b = hp.V_BLK0 + hp.V_NB * g
                val = lambda k, f: self.q(s[b + k], f)  # noqa: E731,B023
                v = c if g == d else 0.25 * sum(val(hp.V_V4 + k, u[g]) for k in (3, 1, 2, 0))
                ul, ur, ull, urr = (val(k, c) for k in (hp.V_UL, hp.V_UR, hp.V_ULL, hp.V_URR))
                bit = lambda k: ((fl >> (4 * g + k)) & 1) == 1  # noqa: E731,B023
                first = first | ~bit(0) | ~bit(1)
                vr, vl = val(hp.V_VCR, u[g]), val(hp.V_VCL, u[g])
                f1 = torch.where(vr > 0, self.cubista(ul, c, ur, vr, true, true), self.cubista(urr, ur, c, vr, bit(3), true))
                f2 = torch.where(vl > 0, self.cubista(ull, ul, c, vl, bit(2), true), self.cubista(ur, c, ul, vl, true, true))
                cub = cub + (f1 - f2) / h
                upw = upw + 0.5 * (v + v.abs()) * (c - ul) / h + 0.5 * (v - v.abs()) * (ur - c) / h
                diff = diff + (ul - 2.0 * c + ur) / (h * h)
                if S is not None:
                    b2 = hp.v_nslot(D, False) + hp.V_NS * g
                    r = [self.q(s[b2 + k], S[d][g]) for k in range(4)]
                    tens = tens + ((r[2] - r[0]) / h if g == d else 0.5 * (r[2] + r[3] - r[0] - r[1]) / (2.0 * h))
            conv = torch.where(first, upw, cub)
            if par["tempdiscrtype"] == hp.SEMI_IMPLICIT_EULER:
                out.append(self.implicit(d, c + par["dt"] * (tens - dp - conv)))
            else:
                out.append(c + par["dt"] * (tens - dp - conv + diff / par["Re"]))
        return out

    def solve(self, b, ops):
        """(c + sum_k A_k) x = b with A_k symmetric along axis k: ops = [A_k], c in ops[-1]."""
        lam, vec = zip(*[torch.linalg.eigh(a) for a in ops[:-1]])
        x, tot = b, ops[-1]
        for k, (l, v) in enumerate(zip(lam, vec)):
            x = torch.movedim(torch.tensordot(v, x, dims=([0], [k])), 0, k)
            tot = tot + l.reshape([-1 if q == k else 1 for q in range(b.dim())])
        if ops[-1] == 0.0:
            flat = tot.reshape(-1)
            at = int(flat.abs().argmin())
            x = x.reshape(-1) / torch.where(torch.arange(len(flat), device=self.dev) == at, math.inf, flat)
            x = x.reshape(b.shape)
        else:
            x = x / tot
        for k, v in enumerate(vec):
            x = torch.movedim(torch.tensordot(v, x, dims=([1], [k])), 0, k)
        return x

    def second(self, m, ends):
        """The 1D second difference over h^2 of m points, diagonal ends as given."""
        a = -2.0 * torch.eye(m, dtype=torch.float64, device=self.dev)
        i = torch.arange(m - 1, device=self.dev)
        a[i, i + 1] = a[i + 1, i] = 1.0
        a[0, 0], a[-1, -1] = ends, ends
        return a / (self.h * self.h)

    def implicit(self, d, rhs):
        r, s = self.par["dt"] / self.par["Re"], self.vs[d]
        # boundary parts of the rows: their values on a zero field
        zero = torch.zeros_like(rhs)
        for g in range(self.D):
            b = hp.V_BLK0 + hp.V_NB * g
            rhs = rhs + r / (self.h * self.h) * (self.q(s[b + hp.V_UL], zero) + self.q(s[b + hp.V_UR], zero))
        dims = [m - (k == d) for k, m in enumerate(self.shape)]
        ops = [-r * self.second(m, -2.0 if k == d else -3.0) for k, m in enumerate(dims)]
        return self.solve(rhs.reshape(dims), ops + [1.0]).reshape(-1)

    def constitutive(self, u, K):
        D, h, par, cs = self.D, self.h, self.par, self.cs
        vl = [self.q(cs[hp.C_BLK0 + hp.C_NB * d + hp.C_UVL], u[d]) for d in range(D)]
        vr = [self.q(cs[hp.C_BLK0 + hp.C_NB * d + hp.C_UVR], u[d]) for d in range(D)]
        Du, pair = [[None] * D for _ in range(D)], 0
        for d in range(D):
            for g in range(D):
                if g == d:
                    Du[d][g] = (vr[d] - vl[d]) / h
                    continue
                q = [self.q(cs[hp.C_BLK0 + hp.C_NB * D + hp.C_NQ * pair + k], u[d]) for k in range(4)]
                pair += 1
                Du[d][g] = (0.25 * (q[3] + vl[d] + vr[d] + q[2]) - 0.25 * (q[1] + vl[d] + vr[d] + q[0])) / h
        M = torch.stack([torch.stack(r, -1) for r in Du], -2)
        Km = torch.stack([torch.stack(r, -1) for r in K], -2)
        l, R = _eigh(Km)
        lam = l.exp()
        Mr = R.mT @ M @ R
        gap = lam[:, None, :] - lam[:, :, None]
        num = Mr * lam[:, None, :] + Mr.mT * lam[:, :, None]
        i, j = torch.triu_indices(D, D, 1, device=self.dev)
        O = torch.zeros_like(Mr)
        O[:, i, j] = num[:, i, j] / (gap[:, i, j] + 1e-12)
        O[:, j, i] = -O[:, i, j]
        O = R @ O @ R.mT
        jl = 1.0 / lam.clamp(min=par["kernel_tol"])
        a = par["alpha"] if par["ve_model"] == hp.GIESEKUS else 0.0
        diag = 2.0 * torch.diagonal(Mr, dim1=1, dim2=2) * lam * jl + ((1 - lam) - a * (1 - lam) ** 2) * jl / par["De"]
        rhs = O @ Km - Km @ O + (R * diag[:, None, :]) @ R.mT
        bit = lambda k: ((self.cf >> k) & 1) == 1  # noqa: E731
        new = [[None] * D for _ in range(D)]
        for i in range(D):
            for j in range(i, D):
                f, conv = K[i][j], 0.0
                for d in range(D):
                    kl, kr, kll, krr = (self.q(cs[hp.C_BLK0 + hp.C_NB * d + k], f) for k in
                                        (hp.C_KL, hp.C_KR, hp.C_KLL, hp.C_KRR))
                    il, ir, ill, irr = (bit(4 * d + k) for k in range(4))
                    conv = conv + self.cell_flux(f, kl, kr, kll, krr, il, ir, ill, irr, vl[d], vr[d]) / h
                new[i][j] = new[j][i] = f + par["dt"] * (rhs[:, i, j] - conv)
        A = _eigh(torch.stack([torch.stack(r, -1) for r in new], -2))
        A = (A[1] * A[0].exp()[:, None, :]) @ A[1].mT
        b, re, de = 1.0 - par["beta"], par["Re"], par["De"]
        S = [[b * A[:, i, j] / (re * de) - b * Du[i][j] / re - (b / (re * de) if i == j else 0.0) for j in range(D)]
             for i in range(D)]
        return new, S

    def cell_flux(self, c, kl, kr, kll, krr, il, ir, ill, irr, vl, vr):
        # right face, then left face; a face whose downwind-side neighbour is
        # outside the domain falls back to upwind on both faces
        f1 = torch.where(vr > 0, self.cubista(kl, c, kr, vr, il, ir), self.cubista(krr, kr, c, vr, irr, ~torch.zeros_like(irr)))
        f2 = torch.where(vl > 0, self.cubista(kll, kl, c, vl, ill, ~torch.zeros_like(ill)), self.cubista(kr, c, kl, vl, ir, il))
        # one cell from the wall the middle branch falls back to upwind too
        f1 = torch.where((vr <= 0) & ~ir, vr * c, f1)
        f2 = torch.where((vr <= 0) & ~ir, torch.where(vl > 0, vl * kl, vl * c), f2)
        left = (vl > 0) & ~il & ~((vr <= 0) & ~ir)
        f1 = torch.where(left, torch.where(vr > 0, vr * c, vr * kr), f1)
        f2 = torch.where(left, vl * c, f2)
        return f1 - f2

    def run(self, fields, steps):
        D, par = self.D, self.par
        u = [self.t(fields[hp.FIELD_U, d]) for d in range(D)]
        p = self.t(fields[hp.FIELD_P, 0])
        ve = self.p.viscoelastic
        K = [[self.t(fields[hp.FIELD_KERNEL, i * D + j]) for j in range(D)] for i in range(D)] if ve else None
        S, pin = None, self.p.pin_row
        lap = [self.second(m, -1.0) for m in self.shape]
        for _ in range(steps):
            if ve:
                K, S = self.constitutive(u, K)
            us = self.velocity(u, p, S)
            b = sum(self.q(self.ds[2 * d + 1], us[d]) - self.q(self.ds[2 * d], us[d]) for d in range(D)) / self.h / par["dt"]
            b[pin] = 0.0
            b[pin] = -b.sum()
            dp = self.solve(b.reshape(self.shape), lap + [0.0]).reshape(-1)
            dp = dp - dp[pin] + (self.p.pin_value - p[pin])
            for d in range(D):
                s = self.vs[d]
                u[d] = us[d] - par["dt"] * (dp[s[hp.V_PR]] - dp[s[hp.V_PL]]) / self.h
            p = p + dp
        out = {f"u{d}": u[d] for d in range(D)}
        out["p"] = p
        if ve:
            out.update({f"K{i}{j}": K[i][j] for i in range(D) for j in range(i, D)})
        return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    parts = _inputs(case, seed)[0]
    limits = [int(x) for x in case["limits"].split(",")] if case["limits"] else [case["steps"]] * len(parts)
    got = [_Exact(p, s, dev).run(f, k) for p, s, f, k in zip(_programs(case), _shapes(case), parts, limits)]
    return {k: torch.cat([g[k] for g in got]).cpu().numpy() for k in got[0]}
