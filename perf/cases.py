"""The work that a user of this library has it do, as cases to be timed.

A case is one call sequence of a user's program on inputs that it holds on the
host: the time loop of a BT-MZ or SP-MZ problem (u in, some steps, u out), the
SSOR iterations of an LU-MZ problem, or the gradient of a BT-MZ or SP-MZ run.
Grids are the NPB-MZ classes S, W, A, B and C of the package's class table;
drawn cases take grids between them, ragged ones among them.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parents[1]
if str(_ROOT / "npbapps.jl_gb300") not in sys.path:
    sys.path.insert(0, str(_ROOT / "npbapps.jl_gb300"))

import npbmz  # noqa: E402
from npbmz import lu  # noqa: E402

VARIANTS = {"fp64": 0, "fp64-graph": npbmz.GRAPH, "exact-graph": npbmz.EXACT | npbmz.GRAPH,
            "mixed-graph": npbmz.MIXED | npbmz.GRAPH, "df-graph": npbmz.MIXED | npbmz.GRAPH | npbmz.RHS_DF}
LU_VARIANTS = {"exact": lu.FACES_NPB | lu.GRAPH, "fma": lu.FACES_NPB | lu.GRAPH | lu.FMA}

# Nominal operations per point and step of the three NPB applications.
FLOPS = {"BT": 3479, "SP": 881, "LU": 1985}


def _class_case(name, kind, cls, variant, steps, **more):
    _, dt, ratio, xz, yz, gx, gy, gz = npbmz.CLASSES[kind][cls]
    case = {"name": name, "work": "steps", "kind": kind, "gx": gx, "gy": gy, "gz": gz, "xz": xz, "yz": yz,
            "ratio": ratio, "dt": dt, "variant": variant, "steps": steps}
    return {**case, **more}


def listed():
    return [
        # the smallest class through the reference's own calls, exch_qbc and adi per step: launches and latency
        _class_case("bt_s_calls", "BT", "S", "fp64", 10, work="calls"),
        # a small run on the refined FP32 sweeps, one graph per step: lines too few to fill the chip
        _class_case("bt_w_mixed", "BT", "W", "mixed-graph", 20),
        # the library's default variant on the middle class
        _class_case("bt_a_fp64", "BT", "A", "fp64", 5),
        # a run that has to match the reference bit for bit
        _class_case("bt_b_exact", "BT", "B", "exact-graph", 2),
        # the benchmark's grid and variant: 256 zones of unequal size, u resident over the steps
        _class_case("bt_c_mixed", "BT", "C", "mixed-graph", 10),
        # the same grid with u kept in the host's own arrays, in and out every step
        _class_case("bt_c_host", "BT", "C", "mixed-graph", 1, work="host"),
        # SP-MZ in FP64, and the large class on the refined FP32 sweeps
        _class_case("sp_b_fp64", "SP", "B", "fp64-graph", 5),
        _class_case("sp_c_mixed", "SP", "C", "mixed-graph", 10),
        # LU-MZ: small, middle (contracted build) and large (bit for bit)
        _class_case("lu_w_exact", "LU", "W", "exact", 10, work="lu"),
        _class_case("lu_b_fma", "LU", "B", "fma", 4, work="lu"),
        _class_case("lu_c_exact", "LU", "C", "exact", 3, work="lu"),
        # the gradient of a run with respect to its forcing and its initial state
        _class_case("bt_w_adjoint", "BT", "W", "fp64", 8, work="adjoint", every=4),
    ]


# dt of the first class whose grid is at least as wide (the class table's own)
def _dt(kind, width):
    if kind == "LU":
        return 1.5e-3 if width < 128 else 2.0
    table = sorted((v[5], v[1]) for v in npbmz.CLASSES[kind].values())
    return next((dt for grid, dt in table if grid >= width), table[-1][1])


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    work = rng.choice(["steps"] * 5 + ["calls", "host", "lu", "lu", "adjoint"])
    kind = "LU" if work == "lu" else rng.choice(["BT", "SP"])
    # zones of 6 to 30 points per side on average (LU-MZ: 8 to 100) and 6 to 28 planes, between class S and class C
    gz = int(_log(rng, 6, 28.99))
    if work == "lu":
        zones = 4
        gx, gy = (zones * int(_log(rng, 8, 100)) for _ in range(2))
        case = {"kind": kind, "gx": gx, "gy": gy, "gz": gz, "xz": zones, "yz": zones, "ratio": 1.0,
                "variant": rng.choice(sorted(LU_VARIANTS))}
    else:
        xz, yz = (rng.choice([2, 4, 8, 16] if work != "adjoint" else [2, 4]) for _ in range(2))
        ratio = rng.choice([1.0, 3.0]) if kind == "BT" else 1.0
        least, most = (6 if ratio == 1.0 else 9), (30 if work != "adjoint" else 18)
        gx, gy = (n * least + int(_log(rng, 1, n * (most - least))) for n in (xz, yz))
        if ratio == 1.0:
            gx, gy = gx // xz * xz, gy // yz * yz
        if work == "calls":
            variant = rng.choice(["fp64", "exact-graph"])
        elif work == "host":
            variant = "mixed-graph"
        elif work == "adjoint":
            variant = "fp64"
        else:
            variant = rng.choice(["fp64", "fp64-graph", "exact-graph", "mixed-graph", "mixed-graph", "df-graph"])
        case = {"kind": kind, "gx": gx, "gy": gy, "gz": gz, "xz": xz, "yz": yz, "ratio": ratio, "variant": variant}
    points = gx * gy * gz
    if points > 4.3e6:  # class C's
        case["gz"] = int(4.3e6 / (gx * gy))
    steps = {"host": 1, "adjoint": 6}.get(work) or max(2, min(10, int(6e6 / points)))
    case.update(work=work, dt=_dt(kind, max(gx, gy)), steps=steps)
    if work == "adjoint":
        case["every"] = 3
    return case


def _points(case):
    return case["gx"] * case["gy"] * case["gz"]


def work(case):
    """Per step u read and written and the forcing read (40 bytes each per point), plus u in and out of the
    host once per call; NPB's operation counts.  A gradient runs each step forward twice and backward once."""
    n, steps = _points(case), case["steps"]
    passes = 3 if case["work"] == "adjoint" else 1
    return {"bytes": n * (80 + 120 * passes * steps), "flops": n * steps * passes * FLOPS[case["kind"]]}


# ---- what a user's program holds before the call --------------------------------------------------------------

def _coefficients(seed):
    """The reference's manufactured-solution table with every coefficient up to 5 % off it."""
    r = np.random.default_rng(seed)
    return npbmz.CE_REFERENCE * r.uniform(0.95, 1.05, (5, 13))


def _geometry(case):
    kind = npbmz.KINDS[case["kind"]]
    dims = [case[k] for k in ("gx", "gy", "gz", "xz", "yz")]
    return npbmz.Geometry(kind, *npbmz.zone_setup(kind, *dims, case["ratio"]), *dims)


def prepare(case, seed):
    if case["work"] == "lu":
        nx, ny, nz, nbr = lu.lu_zone_setup(case["gx"], case["gy"], case["gz"], case["xz"], case["yz"], case["ratio"])
        p = lu.LuProblem(nx, ny, nz, nbr, case["dt"], flags=LU_VARIANTS[case["variant"]])
        p.setup(_coefficients(seed))
        fields = [torch.zeros(5 * p.points, dtype=torch.float64).pin_memory() for _ in range(4)]
        for t, field in zip(fields, (lu.U, lu.RSD)):
            p.download(-1, field, out=t.numpy())
        return {"case": case, "p": p, "u": fields[0], "rsd": fields[1], "u_out": fields[2], "rsd_out": fields[3]}
    p = npbmz.Problem(_geometry(case), case["dt"], VARIANTS[case["variant"]])
    p.setup(_coefficients(seed))
    layout, n = npbmz.LAYOUT_DENSE, p.dense_total()
    if case["work"] == "host":
        layout = npbmz.LAYOUT_REF
        g = p.geom
        n = sum(npbmz.ref_elems(g.kind, npbmz.U, int(a), int(b), int(c)) for a, b, c in zip(g.nx, g.ny, g.nz))
    u = torch.zeros(n, dtype=torch.float64).pin_memory()
    p.transfer_raw(npbmz.U, -1, layout, u.data_ptr(), False)
    s = {"case": case, "p": p, "u": u, "layout": layout}
    if case["work"] == "adjoint":
        noise = np.random.default_rng(seed + 1).normal(0.0, 0.01, n)
        s["target"] = u.numpy() + noise
    elif case["work"] != "host":
        s["out"] = torch.zeros(n, dtype=torch.float64).pin_memory()
    return s


def run(s):
    case, p = s["case"], s["p"]
    if case["work"] == "lu":
        p.upload(-1, lu.U, s["u"].numpy())
        p.upload(-1, lu.RSD, s["rsd"].numpy())
        p.iterate(case["steps"])
        p.download(-1, lu.U, out=s["u_out"].numpy())
        p.download(-1, lu.RSD, out=s["rsd_out"].numpy())
        return s["u_out"], s["rsd_out"]
    if case["work"] == "adjoint":
        objective, forcing, u0 = p.adjoint(case["steps"], s["target"], checkpoint_every=case["every"])
        return objective, p.flatten(forcing), p.flatten(u0)
    if case["work"] == "host":  # u stays in the caller's arrays, as in the reference's loop
        p.step_inout(case["steps"], s["layout"], s["u"].data_ptr(), s["u"].data_ptr())
        return s["u"]
    if case["work"] == "calls":
        p.transfer_raw(npbmz.U, -1, s["layout"], s["u"].data_ptr(), True)
        for _ in range(case["steps"]):
            npbmz.exch_qbc(p)
            npbmz.adi(p)
        p.transfer_raw(npbmz.U, -1, s["layout"], s["out"].data_ptr(), False)
        return s["out"]
    p.step_inout(case["steps"], s["layout"], s["u"].data_ptr(), s["out"].data_ptr())
    return s["out"]


# ---- the same in plain torch, 64 bits --------------------------------------------------------------------------
# Fields are [5, zone, k, j, i], every zone padded to the largest; direction 0, 1, 2 is the axis i, j, k.

C1, C2, C3C4, C1C5, C1345, CON43 = 1.4, 0.4, 0.1, 1.96, 0.196, 4.0 / 3.0
AXIS = (4, 3, 2)
D = (0.75, 0.75, 1.0)
DSSP = 0.25
STENCILS = ((0, 0, 5, -4, 1), (0, -4, 6, -4, 1), (1, -4, 6, -4, 1), (1, -4, 6, -4, 0), (1, -4, 5, 0, 0))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _shift(a, by, axis):
    return torch.roll(a, -by, axis)


class _Zones:
    """Padded fields of the zones, masks of their interiors, the dissipation's weights and the face copies."""

    def __init__(self, nx, ny, nz, nbr, lu_faces=False):
        self.n = [np.asarray(v, np.int64) for v in (nx, ny, nz)]
        self.count, self.size = len(nx), [int(v.max()) for v in self.n]
        self.shape = (self.count, self.size[2], self.size[1], self.size[0])
        dev = _device()
        self.line, self.weights = [], []
        for d in range(3):
            q = np.arange(self.size[d])[None, :]
            n = self.n[d][:, None]
            classes = (q == 1, q == 2, (q >= 3) & (q <= n - 4), q == n - 3, q == n - 2)
            w = sum(np.asarray(c, float)[..., None] * np.asarray(s, float) for c, s in zip(classes, STENCILS))
            at = [self.count, 1, 1, 1]
            at[AXIS[d] - 1] = self.size[d]
            self.line.append(torch.tensor((q >= 1) & (q <= n - 2), device=dev))
            self.weights.append([torch.tensor(w[..., o], device=dev).reshape(at) for o in range(5)])
        x, y, z = self.line
        self.inside = z[:, :, None, None] & y[:, None, :, None] & x[:, None, None, :]
        src, dst = [], []
        point = np.arange(int(np.prod(self.shape))).reshape(self.shape)
        for a in range(self.count):
            w, e, s, n = (int(v) for v in nbr[4 * a:4 * a + 4])
            (ax, ay, az), k = (int(v[a]) for v in self.n), slice(1, int(self.n[2][a]) - 1)
            if lu_faces:  # west / east step along j there and own the corners
                faces = [((a, k, 0, slice(0, ax)), (w, k, int(self.n[1][w]) - 2, slice(0, ax))),
                         ((a, k, ay - 1, slice(0, ax)), (e, k, 1, slice(0, ax))),
                         ((a, k, slice(1, ay - 1), 0), (n, k, slice(1, ay - 1), int(self.n[0][n]) - 2)),
                         ((a, k, slice(1, ay - 1), ax - 1), (s, k, slice(1, ay - 1), 1))]
            else:
                j, i = slice(1, ay - 1), slice(1, ax - 1)
                faces = [((a, k, j, 0), (w, k, j, int(self.n[0][w]) - 2)), ((a, k, j, ax - 1), (e, k, j, 1)),
                         ((a, k, 0, i), (s, k, int(self.n[1][s]) - 2, i)), ((a, k, ay - 1, i), (n, k, 1, i))]
            for to, of in faces:
                dst.append(point[to].reshape(-1))
                src.append(point[of].reshape(-1))
        self.src, self.dst = (torch.tensor(np.concatenate(v), device=dev) for v in (src, dst))

    def pad(self, flat, rest=(1.0, 0.0, 0.0, 0.0, 1.0)):
        f = torch.as_tensor(flat, device=_device())
        out = torch.tensor(rest, dtype=torch.float64, device=f.device).reshape(5, 1, 1, 1, 1).repeat(1, *self.shape)
        at = 0
        for a in range(self.count):
            x, y, z = (int(v[a]) for v in self.n)
            out[:, a, :z, :y, :x] = f[at:at + 5 * x * y * z].reshape(5, z, y, x)
            at += 5 * x * y * z
        return out

    def flat(self, field):
        return torch.cat([field[:, a, :int(self.n[2][a]), :int(self.n[1][a]), :int(self.n[0][a])].reshape(-1)
                          for a in range(self.count)]).detach()

    def exchange(self, u):
        if self.count < 2:
            return u
        v = u.reshape(5, -1)
        return v.index_copy(1, self.dst, v[:, self.src]).reshape(u.shape)


def _state(u):
    ri = 1.0 / u[0]
    vel = u[1:4] * ri
    return ri, vel, 0.5 * (vel * vel).sum(0), u[4] * ri


def _convective(u, d):
    _, vel, q, _ = _state(u)
    p = C2 * (u[4] - q * u[0])
    f = [u[1 + d]] + [u[m + 1] * vel[d] + (p if m == d else 0.0) for m in range(3)]
    return torch.stack(f + [(C1 * u[4] - C2 * q * u[0]) * vel[d]])


def _jacobians(u, d):
    """d(convective flux) / du and d(viscous flux) / du of direction d at states u [5, ...], as [..., 5, 5]."""
    ri, vel, q, e = _state(u)
    vn, zero, one = vel[d], torch.zeros_like(ri), torch.ones_like(ri)
    f, n = [[zero] * 5 for _ in range(5)], [[zero] * 5 for _ in range(5)]
    f[0][1 + d] = one
    n[4][0], n[4][4] = -C1345 * e * ri, C1345 * ri
    for m in range(3):
        c = C3C4 * (CON43 if m == d else 1.0)
        n[m + 1][0], n[m + 1][m + 1] = -c * ri * vel[m], c * ri
        n[4][0] = n[4][0] - (c - C1345) * ri * vel[m] * vel[m]
        n[4][m + 1] = (c - C1345) * ri * vel[m]
        if m == d:
            f[m + 1][0] = C2 * q - vn * vn
            f[m + 1][1 + d], f[m + 1][4] = (2.0 - C2) * vn, C2 * one
        else:
            f[m + 1][0], f[m + 1][m + 1], f[m + 1][1 + d] = -vel[m] * vn, vn, vel[m]
            f[1 + d][m + 1] = -C2 * vel[m]
            f[4][m + 1] = -C2 * vel[m] * vn
    f[4][0] = (2.0 * C2 * q - C1 * e) * vn
    f[4][1 + d], f[4][4] = C1 * e - C2 * (q + vn * vn), C1 * vn
    return tuple(torch.stack([torch.stack(row, -1) for row in a], -2) for a in (f, n))


def _operator(z, u, t1, t2, t3):
    """The spatial operator of the three applications, without the forcing: -dF/dx + viscous terms + dissipation."""
    _, vel, q, e = _state(u)
    total = torch.zeros_like(u)
    for d in range(3):
        ax = AXIS[d]

        def second(a):
            return _shift(a, 1, ax - 1) - 2.0 * a + _shift(a, -1, ax - 1)

        f = _convective(u, d)
        visc = [torch.zeros_like(q)] + [(CON43 if m == d else 1.0) * second(vel[m]) for m in range(3)]
        visc.append((1.0 - C1C5) * second(q) + second(vel[d] * vel[d]) / 6.0 + C1C5 * second(e))
        rough = sum(w * _shift(u, o - 2, ax) for o, w in enumerate(z.weights[d]))
        total = total - t2[d] * (_shift(f, 1, ax) - _shift(f, -1, ax)) + C3C4 * t3[d] * t3[d] * torch.stack(visc)
        total = total + D[d] * t1[d] * (_shift(u, 1, ax) - 2.0 * u + _shift(u, -1, ax)) - DSSP * rough
    return total


def _lines(z, a, d):
    """Field a [5, zone, k, j, i] as interior lines along d: [point, zone, transverse, transverse, 5]."""
    a = a.movedim(0, -1).movedim(AXIS[d] - 1, 0)
    return a[:, :, 1:-1, 1:-1]


def _put_lines(z, a, x, d):
    """a with the lines x of direction d in the place of its interior points."""
    full = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1)).movedim(0, AXIS[d] - 1).movedim(-1, 0)
    return torch.where(z.inside, full, a)


def _bt_solve(z, u, r, d, dt, t1, t2):
    U, R, eye = _lines(z, u, d), _lines(z, r, d), torch.eye(5, dtype=torch.float64, device=u.device)
    n, t1, t2 = U.shape[0], dt * t1[d], dt * t2[d]

    def at(p):
        f, v = _jacobians(U[p].movedim(-1, 0), d)
        return t2 * f, t1 * (v + D[d] * eye)

    back, now = at(0), at(1)
    C, x = [torch.zeros_like(back[0])], [R[0]]
    for p in range(1, n - 1):
        ahead = at(p + 1)
        on = z.line[d][:, p].reshape(-1, 1, 1, 1, 1).double()
        A, B, Cp = -(back[0] + back[1]) * on, eye + 2.0 * now[1] * on, (ahead[0] - ahead[1]) * on
        rhs = R[p][..., None] - A @ x[-1][..., None]
        s = torch.linalg.solve(B - A @ C[-1], torch.cat([Cp, rhs], -1))
        C.append(s[..., :5])
        x.append(s[..., 5])
        back, now = now, ahead
    x.append(R[n - 1])
    for p in range(n - 2, 0, -1):
        x[p] = x[p] - (C[p] @ x[p + 1][..., None])[..., 0]
    return _put_lines(z, r, torch.stack(x), d)


def _sp_solve(z, u, r, d, dt, t1, t2):
    U, R = _lines(z, u, d).movedim(-1, 0), _lines(z, r, d)
    n, a1, a2, comz = U.shape[1], dt * t1[d], dt * t2[d], dt * DSSP
    ri, vel, q, e = _state(U)
    ru = C3C4 * ri
    rhon = torch.maximum(torch.maximum(D[d] + CON43 * ru, D[d] + C1C5 * ru), torch.maximum(D[d] + ru, 0.0 * ru + D[d]))
    sound, cv = torch.sqrt(C1 * C2 * (e - q)), vel[d]
    rows = []
    for p in range(n):
        b, a = max(p - 1, 0), min(p + 1, n - 1)
        on = z.line[d][:, p].reshape(-1, 1, 1).double()
        w = [z.weights[d][o].reshape(z.count, -1)[:, p].reshape(-1, 1, 1) * comz for o in range(5)]
        per = []
        for c in (0.0, 1.0, -1.0):  # the three systems: the flow's speed, and the speed of sound either way
            per.append(torch.stack([w[0] + 0.0 * ri[p], w[1] - a2 * (cv[b] + c * sound[b]) - a1 * rhon[b],
                                    w[2] + 2.0 * a1 * rhon[p], w[3] + a2 * (cv[a] + c * sound[a]) - a1 * rhon[a],
                                    w[4] + 0.0 * ri[p]]) * on)
        L = torch.stack([per[0], per[0], per[0], per[1], per[2]], -1)
        rows.append([L[0], L[1], 1.0 + L[2], L[3], L[4]])
    x = [R[p] for p in range(n)]
    for p in range(n):
        s = 1.0 / rows[p][2]
        rows[p][3], rows[p][4], x[p] = rows[p][3] * s, rows[p][4] * s, x[p] * s
        if p + 1 < n:
            m = rows[p + 1][1]
            rows[p + 1][2], rows[p + 1][3] = rows[p + 1][2] - m * rows[p][3], rows[p + 1][3] - m * rows[p][4]
            x[p + 1] = x[p + 1] - m * x[p]
        if p + 2 < n:
            m = rows[p + 2][0]
            rows[p + 2][1], rows[p + 2][2] = rows[p + 2][1] - m * rows[p][3], rows[p + 2][2] - m * rows[p][4]
            x[p + 2] = x[p + 2] - m * x[p]
    for p in range(n - 2, -1, -1):
        x[p] = x[p] - rows[p][3] * x[p + 1] - (rows[p][4] * x[p + 2] if p + 2 < n else 0.0)
    v = _put_lines(z, r, torch.stack(x), d)
    bt, half = math.sqrt(0.5), 0.5 * (v[3] + v[4])
    if d == 0:
        o = [-v[1], v[0], bt * (v[3] - v[4]), half - bt * v[2], half + bt * v[2]]
    elif d == 1:
        o = [bt * (v[3] - v[4]), -v[2], v[1], half - bt * v[0], half + bt * v[0]]
    else:
        ri, w, q, e = _state(u)
        ac, b = torch.sqrt(C1 * C2 * (e - q)), bt * u[0]
        s, m = b / ac * (v[3] + v[4]), b * (v[3] - v[4])
        t = v[2] + s
        o = [t, w[0] * t - u[0] * v[1], u[0] * v[0] + w[1] * t, w[2] * t + m,
             u[0] * (w[1] * v[0] - w[0] * v[1]) + q * t + 2.5 * ac * ac * s + w[2] * m]
    return torch.where(z.inside, torch.stack(o), v)


def _txinvr(u, r):
    ri, w, q, e = _state(u)
    ac, bt = torch.sqrt(C1 * C2 * (e - q)), math.sqrt(0.5)
    s = C2 / (ac * ac) * (q * r[0] - w[0] * r[1] - w[1] * r[2] - w[2] * r[3] + r[4])
    t, m = bt * ri * (w[0] * r[0] - r[1]), bt * ri * ac * s
    return torch.stack([r[0] - s, ri * (r[3] - w[2] * r[0]), ri * (w[1] * r[0] - r[2]), m - t, m + t])


def _step(z, case, u, forcing):
    h = [(case["gx"] - 1) / case["xz"], (case["gy"] - 1) / case["yz"], float(case["gz"] - 1)]
    t1, t2, dt = [v * v for v in h], [0.5 * v for v in h], case["dt"]
    u = z.exchange(u)
    r = dt * (forcing + _operator(z, u, t1, t2, h))
    r = torch.where(z.inside, _txinvr(u, r) if case["kind"] == "SP" else r, forcing)
    for d in range(3):
        r = (_sp_solve if case["kind"] == "SP" else _bt_solve)(z, u, r, d, dt, t1, t2)
    return torch.where(z.inside, u + r, u)


def _lu_iterations(case, z, u, rsd, frct, omega):
    nx, ny, nz = z.size
    h = [nx - 1.0, ny - 1.0, nz - 1.0]
    t1, t2, dt = [v * v for v in h], [0.5 * v for v in h], case["dt"]
    dev, eye = u.device, torch.eye(5, dtype=torch.float64, device=u.device)
    off = (1, nx, nx * ny)
    k, j, i = np.meshgrid(np.arange(1, nz - 1), np.arange(1, ny - 1), np.arange(1, nx - 1), indexing="ij")
    level, point = (i + j + k).reshape(-1), ((k * ny + j) * nx + i).reshape(-1)
    planes = [torch.tensor(point[level == v], device=dev) for v in range(3, level.max() + 1)]
    for _ in range(case["steps"]):
        u = z.exchange(u)
        states = u.reshape(5, z.count, -1)
        w = torch.where(z.inside, dt * rsd, rsd).reshape(5, z.count, -1).permute(1, 2, 0).contiguous()
        low, up, diag = [], [], eye
        for d in range(3):
            f, v = _jacobians(states, d)
            v = dt * t1[d] * (v + D[d] * eye)
            low.append(-dt * t2[d] * f - v)
            up.append(dt * t2[d] * f - v)
            diag = diag + 2.0 * v
        diag = torch.linalg.inv(diag)

        def near(blocks, at, sign):
            return sum((blocks[d][:, at + sign * off[d]] @ w[:, at + sign * off[d]][..., None])[..., 0]
                       for d in (2, 1, 0))

        for at in planes:
            w[:, at] = (diag[:, at] @ (w[:, at] - omega * near(low, at, -1))[..., None])[..., 0]
        for at in reversed(planes):
            w[:, at] = w[:, at] - (diag[:, at] @ (omega * near(up, at, 1))[..., None])[..., 0]
        r = w.permute(2, 0, 1).reshape(u.shape)
        u = torch.where(z.inside, u + r / (omega * (2.0 - omega)), u)
        rsd = torch.where(z.inside, _operator(z, u, t1, t2, h) - frct, -frct)
    return u, rsd


def _reference_layout(z, u, kind):
    """u in the reference's own array of every zone, its halo left at zero."""
    out = []
    for a in range(z.count):
        x, y, n = (int(v[a]) for v in z.n)
        part = u[:, a, :n, :y, :x]
        if kind == "BT":
            full = torch.zeros(n + 5, y + 5, x + 5, 5, dtype=torch.float64, device=u.device)
            full[2:2 + n, 2:2 + y, 2:2 + x] = part.movedim(0, -1)
        else:
            full = torch.zeros(5, n + 5, (y + 1) // 2 * 2 + 5, (x + 1) // 2 * 2 + 5, dtype=torch.float64, device=u.device)
            full[:, 2:2 + n, 2:2 + y, 2:2 + x] = part
        out.append(full.reshape(-1))
    return torch.cat(out)


def exact(case, seed):
    s = prepare(case, seed)
    p = s["p"]
    if case["work"] == "lu":
        z = _Zones(p.nx, p.ny, p.nz, p.nbr, lu_faces=True)
        u, rsd = z.pad(s["u"]), z.pad(s["rsd"], (0.0,) * 5)
        frct = torch.zeros_like(s["u"])
        p.download(-1, lu.FRCT, out=frct.numpy())
        u, rsd = _lu_iterations(case, z, u, rsd, z.pad(frct, (0.0,) * 5), p.omega)
        return z.flat(u), z.flat(rsd)
    g = p.geom
    z = _Zones(g.nx, g.ny, g.nz, g.nbr)
    dense = np.zeros(p.dense_total())
    p.transfer_raw(npbmz.U, -1, npbmz.LAYOUT_DENSE, dense.ctypes.data, False)
    forcing = z.pad(np.concatenate([f.reshape(-1) for f in p.download_all(npbmz.FORCING)]), (0.0,) * 5)
    u = z.pad(dense)
    if case["work"] == "adjoint":
        u.requires_grad_(True)
        forcing.requires_grad_(True)
        v = u
        for _ in range(case["steps"]):
            v = _step(z, case, v, forcing)
        # padding points differ from no target: they add nothing
        target = z.pad(s["target"])
        objective = 0.5 * ((v - target) ** 2).sum()
        objective.backward()
        return objective.detach(), z.flat(forcing.grad), z.flat(u.grad)
    for _ in range(case["steps"]):
        u = _step(z, case, u, forcing)
    return _reference_layout(z, u, case["kind"]) if case["work"] == "host" else z.flat(u)
