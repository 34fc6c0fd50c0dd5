"""The work that users of this package give it, as cases to be timed.

Four kinds of call, each through the public entry points:

  rhs    one inviscid right-hand side by the drop-in sequence of a host code that owns its
         fields: ghost fill of d, u, v, w, T, sound speed, du
  loop   one SSP-RK3 step of such a host code: three times ghost fill, sound speed, du,
         stage update, conserved to primitive
  step   one SSP-RK3 step of a device-resident Solver (Euler, or Navier-Stokes with CD6 / CD8
         viscous terms)
  batch  a Batch of uneven grids taken `steps` steps, and every grid's state fetched

over both precisions, periodic, zero-gradient and CLOSURE faces, Cartesian and general
metrics.  `exact` evaluates the same scheme in 64 bits with torch alone: Steger-Warming
splitting, the WENO7-SYMBO reconstruction written on the stencil values, the WENO5-type
closures, central differences.
"""
import math
import random

import numpy as np
import torch

import windstencil_b200 as ws

GAMMA, EPSL = 1.4, 1e-6
FACES = {
    "periodic": (ws.FACE_PERIODIC,) * 6,
    "outflow": (ws.FACE_EXTRAP,) * 2 + (ws.FACE_PERIODIC,) * 4,       # a shock tube along x
    "closure": (ws.FACE_CLOSURE,) * 4 + (ws.FACE_PERIODIC,) * 2,      # walls in x and y
}
FLOP_RHS = 7266.0        # operations per cell of one inviscid RHS (sqrt and divide count 1)
FLOP_VIS = 330.0         # of the viscous terms (CD8; CD6 somewhat fewer)


def listed():
    return [
        # the smallest grid that the benchmark configurations name: latency and launches count
        case("rhs", 64, 32, 16, name="rhs_small"),
        # the headline grid, Sod jump along x, as a host code calls it once per stage
        case("rhs", 600, 128, 128, faces="outflow", flow="sod", name="rhs_large"),
        # a curvilinear mesh of odd extents: general metrics at every point
        case("rhs", 157, 93, 61, metrics=True, name="rhs_metrics"),
        # the mixed form through the drop-in entry, the smallest grid of the published tables
        case("rhs", 480, 64, 32, precision="mixed", faces="outflow", flow="sod", name="rhs_mixed"),
        # a whole RK3 step of a host code that keeps its own fields, odd extents
        case("loop", 201, 101, 67, name="loop_odd"),
        # solver steps: smallest, largest in both precisions
        case("step", 64, 32, 16, name="step_small"),
        case("step", 600, 128, 128, faces="outflow", flow="sod", name="step_large"),
        case("step", 600, 128, 128, precision="mixed", name="step_mixed_large"),
        # walls in x and y by the reference's boundary closures
        case("step", 240, 96, 72, faces="closure", flow="sod", name="step_closure"),
        # Navier-Stokes with 8th-order viscous derivatives
        case("step", 300, 128, 64, viscous=8, name="step_navier_stokes"),
        # many uneven grids advanced together and fetched, FP64 and mixed
        case("batch", 0, 0, 0, grids=12, steps=20, name="batch_fp64"),
        case("batch", 0, 0, 0, precision="mixed", grids=32, steps=50, name="batch_mixed"),
    ]


def case(kind, nx, ny, nz, precision="fp64", faces="periodic", flow="fourier", metrics=False,
         viscous=0, grids=0, steps=1, name=None):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, faces=faces, flow=flow,
             metrics=metrics, viscous=viscous, grids=grids, steps=steps)
    if name:
        c["name"] = name
    return c


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["rhs", "rhs", "loop", "step", "step", "step", "batch"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "batch":
        return case(kind, 0, 0, 0, precision, grids=rng.randint(4, 16), steps=rng.randint(8, 30))
    nx, ny, nz = _extent(rng, 16, 600), _extent(rng, 12, 200), _extent(rng, 12, 160)
    flow = rng.choice(["fourier", "sod"])
    if kind == "rhs" and rng.random() < 0.4:
        nx, ny, nz = min(nx, 300), min(ny, 128), min(nz, 96)
        return case(kind, nx, ny, nz, precision, metrics=True)
    faces = rng.choice(["periodic", "outflow", "closure"])
    viscous = rng.choice([0, 0, 6, 8]) if kind == "step" and faces != "closure" else 0
    return case(kind, nx, ny, nz, precision, faces, flow, viscous=viscous)


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _modes(gen, nx, ny, nz, dev, nmodes=8, amp=0.05):
    """Sum of nmodes Fourier modes of wavenumbers 1..4, amplitudes up to amp."""
    k = torch.randint(1, 5, (nmodes, 3), generator=gen).double()
    a = torch.rand(nmodes, generator=gen, dtype=torch.float64) * amp
    ph = torch.rand(nmodes, generator=gen, dtype=torch.float64) * 2 * math.pi
    out = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
    x, y, z = (2 * math.pi / n * torch.arange(n, dtype=torch.float64) for n in (nx, ny, nz))
    for m in range(nmodes):
        ex, ey = torch.polar(torch.ones(nx).double(), k[m, 0] * x), torch.polar(
            torch.ones(ny).double(), k[m, 1] * y)
        ez = torch.polar(torch.ones(nz).double(), k[m, 2] * z + ph[m])
        yz = (ez[:, None] * ey[None, :]).to(dev)
        ex = ex.to(dev)
        out += a[m] * (yz.imag[:, :, None] * ex.real + yz.real[:, :, None] * ex.imag)
    return out


def _state(nx, ny, nz, flow, seed, dev):
    """Primitives d, u, v, w, T: a smooth Mach 0.5 flow with a contact, or a Sod jump with 1%
    noise."""
    gen = torch.Generator().manual_seed(seed)
    x = torch.arange(nx, dtype=torch.float64, device=dev)
    if flow == "fourier":
        d = 1.0 + _modes(gen, nx, ny, nz, dev)
        d = d * (1.0 + (x * 2 > nx).double())
        u = 0.5 + _modes(gen, nx, ny, nz, dev)
        v, w = _modes(gen, nx, ny, nz, dev), _modes(gen, nx, ny, nz, dev)
        T = 1.0 / d
    else:
        gd = torch.Generator(device=dev).manual_seed(seed)
        jump = 0.3 + 0.4 * float(torch.rand(1, generator=gen))

        def noise():
            return 0.01 * (2 * torch.rand((nz, ny, nx), generator=gd, dtype=torch.float64,
                                          device=dev) - 1)
        left = (x + 0.5 < jump * nx).double()
        d = (0.125 + 0.875 * left) * (1.0 + noise())
        u, v, w = torch.zeros_like(d), noise(), noise()
        T = GAMMA * (0.1 + 0.9 * left) / d
    return d, u, v, w, T


def _cons(p):
    d, u, v, w, T = p
    cv = 1.0 / (GAMMA * (GAMMA - 1.0))
    return torch.stack([d, u * d, v * d, w * d, d * ((u * u + v * v + w * w) * 0.5 + cv * T)])


def _metric_fields(g, seed, dev):
    """akx..asz and J on the padded points of a smoothly sheared mesh, with its ghost values."""
    gen = torch.Generator().manual_seed(seed + 101)
    z, y, x = torch.meshgrid(*(torch.linspace(0, 2 * math.pi, n + 8, dtype=torch.float64)
                               for n in (g.nz, g.ny, g.nx)), indexing="ij")
    out = []
    for i in range(10):
        a, b, c = (float(t) for t in torch.rand(3, generator=gen) * 2 * math.pi)
        wave = torch.sin(x + a) * torch.cos(y + b) + 0.5 * torch.sin(z + c)
        out.append(((1.0 if i % 4 == 0 or i == 9 else 0.0) + 0.15 * wave).to(dev))
    return out


def _grids(c, seed):
    """(nx, ny, nz, mode seed) of the batch's grids: nx in [32, 256], ny, nz in [16, 128]."""
    r = random.Random(c["grids"] * 1000 + c["steps"])
    return [(_extent(r, 32, 256), _extent(r, 16, 128), _extent(r, 16, 128), 1000 * seed + i)
            for i in range(c["grids"])]


def _grid(c, nx=None, ny=None, nz=None):
    return ws.Grid(nx or c["nx"], ny or c["ny"], nz or c["nz"], faces=FACES[c["faces"]],
                   precision=ws.MIXED if c["precision"] == "mixed" else ws.FP64,
                   metrics_uniform=not c["metrics"])


VIS = dict(re=1e4, pr=0.72, ref_t=288.15)


def prepare(c, seed):
    dev = "cuda"
    if c["kind"] == "batch":
        specs = _grids(c, seed)
        b = ws.Batch([_grid(c, *s[:3]) for s in specs])
        for i, s in enumerate(specs):
            b.set_state(i, _cons(_state(*s[:3], c["flow"], s[3], dev)).cpu().numpy())
        b.set_dt(b.compute_dt(0.4))
        return {"c": c, "batch": b, "n": len(specs)}
    g = _grid(c)
    prims = _state(g.nx, g.ny, g.nz, c["flow"], seed, dev)
    if c["kind"] == "step":
        s = ws.Solver(g)
        s.set_state(_cons(prims).cpu().numpy())
        if c["viscous"]:
            s.set_viscous(dict(VIS, scheme=c["viscous"]))
        torch.cuda.synchronize()
        return {"c": c, "g": g, "solver": s, "dt": s.compute_dt(0.4)}
    fields = []
    for p in prims:
        t = ws.lap_tensor(g)
        t[4:4 + g.nz, 4:4 + g.ny, 4:4 + g.nx] = p
        fields.append(t)
    st = {"c": c, "g": g, "job": ws.interior_job(g), "fields": fields, "cc": ws.lap_tensor(g),
          "du": ws.soa_tensor(g), "met": None}
    if c["metrics"]:
        st["met"] = []
        for m in _metric_fields(g, seed, dev):
            t = ws.lap_tensor(g)
            t[:, :, :g.nx + 8] = m
            st["met"].append(t)
    if c["kind"] == "loop":
        st["f"], st["fn"] = _cons(prims).contiguous(), ws.soa_tensor(g)
        st["dt"] = 0.4 / _max_speed(g, prims)
    return st


class _View:
    """A Solver's device field as torch sees it; the tensor made of it keeps the Solver, which
    owns the memory."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": None,
                                         "typestr": "<f8", "version": 3}


def _du(st):
    d, u, v, w, T = st["fields"]
    ws.ghost_fill(st["g"], st["fields"])
    ws.du_invis_jacobian3d_init(st["g"], st["job"], T, st["cc"])
    ws.du_invis_jacobian3d(st["g"], st["job"], d, u, v, w, st["cc"], st["du"], metrics=st["met"])


def run(st):
    c = st["c"]
    if c["kind"] == "rhs":
        _du(st)
        return st["du"]
    if c["kind"] == "loop":
        st["fn"].copy_(st["f"])
        for krk in (1, 2, 3):
            _du(st)
            ws.time_advance(st["g"], krk, st["dt"], st["f"], st["fn"], st["du"])
            ws.cons_to_prim(st["g"], st["f"], *st["fields"])
        return st["f"]
    if c["kind"] == "step":
        s, g = st["solver"], st["g"]
        s.step(st["dt"], c["steps"])
        f = s.fields()[0]
        return torch.as_tensor(_View(s, f.ptr, (5, g.nz, g.ny, g.nx)), device="cuda")
    st["batch"].step(c["steps"])
    return [st["batch"].get_state(i) for i in range(st["n"])]


def work(c):
    """Bytes: each input field read once and each output written once; operations of the
    scheme as it is written."""
    if c["kind"] == "batch":
        cells = sum(s[0] * s[1] * s[2] for s in _grids(c, 0))
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    per = 80.0 + (80.0 if c["metrics"] else 0.0)     # state or primitives in, state or du out
    rhs = 1 if c["kind"] == "rhs" else 3 * c["steps"]
    flops = (FLOP_RHS + (FLOP_VIS if c["viscous"] else 0.0)) * rhs
    # the fetched states of a batch leave the device once, whatever the number of steps
    return {"bytes": per * cells * (1 if c["kind"] in ("rhs", "loop") else c["steps"]),
            "flops": flops * cells}


def tolerance(c):
    """Relative differences that another evaluation order shows, about four times what the
    path differs by from `exact`: in du FP64 rounding amplified by the differences over h (6e-15
    to 9e-15 measured) or the FP32 rounding of the split fluxes (2e-6); a step multiplies them
    by dt (1.4e-16, 1.8e-8), and many steps let them grow (8e-16 after 20)."""
    fp64 = c["precision"] == "fp64"
    if c["kind"] == "rhs":
        return {"rel": 4e-14, "max": 4e-12} if fp64 else {"rel": 1e-5, "max": 1e-3}
    if c["kind"] == "batch":
        return {"rel": 1e-14, "max": 1e-12} if fp64 else {"rel": 2e-6, "max": 2e-4}
    return {"rel": 2e-15, "max": 2e-13} if fp64 else {"rel": 1e-7, "max": 1e-5}


# ---------------------------------------------------------------------------------------
# the same scheme in 64 bits, by torch alone
# ---------------------------------------------------------------------------------------
def _max_speed(g, p):
    d, u, v, w, T = p
    rx, ry, rz = 1 / g.hx, 1 / g.hy, 1 / g.hz
    return float((u.abs() * rx + v.abs() * ry + w.abs() * rz +
                  T.sqrt() * math.sqrt(rx * rx + ry * ry + rz * rz)).max())


def _extend(p, kinds, axis):
    """Four ghost points on both sides along `axis` (0 x, 1 y, 2 z)."""
    dim = 2 - axis + (p.dim() - 3)
    n = p.shape[dim]
    idx = torch.arange(-4, n + 4, device=p.device)
    lo, hi = kinds[2 * axis], kinds[2 * axis + 1]
    src = idx.clone()
    src[:4] = idx[:4] + n if lo == ws.FACE_PERIODIC else 0
    src[-4:] = idx[-4:] - n if hi == ws.FACE_PERIODIC else n - 1
    return p.index_select(dim, src)


def _split(p, cc, a):
    """Steger-Warming F+ and F- (stacked over the five variables); a: metric gradient."""
    d, u, v, w = p
    a1, a2, a3 = a
    ss = (a1 * a1 + a2 * a2 + a3 * a3) ** 0.5
    k1, k2, k3 = a1 / ss, a2 / ss, a3 / ss
    e1 = a1 * u + a2 * v + a3 * w
    e2, e3 = e1 - cc * ss, e1 + cc * ss
    plus = [(e + (e * e + EPSL * EPSL).sqrt()) * 0.5 for e in (e1, e2, e3)]
    t0 = d / (2 * GAMMA)
    u1, v1, w1, u2, v2, w2 = (u - cc * k1, v - cc * k2, w - cc * k3, u + cc * k1, v + cc * k2,
                              w + cc * k3)
    q1, q2 = (u1 * u1 + v1 * v1 + w1 * w1) * 0.5, (u2 * u2 + v2 * v2 + w2 * w2) * 0.5
    vv = (GAMMA - 1) * (u * u + v * v + w * w)
    ww = (3 - GAMMA) / (2 * (GAMMA - 1)) * cc * cc
    out = []
    for x1, x2, x3 in (plus, [e - q for e, q in zip((e1, e2, e3), plus)]):
        c1 = 2 * (GAMMA - 1) * x1
        out.append(torch.stack([t0 * (c1 + x2 + x3), t0 * (c1 * u + x2 * u1 + x3 * u2),
                                t0 * (c1 * v + x2 * v1 + x3 * v2),
                                t0 * (c1 * w + x2 * w1 + x3 * w2),
                                t0 * (x1 * vv + x2 * q1 + x3 * q2 + ww * (x2 + x3))]))
    return out


_D = (0.0401954833730, 0.2493800006710, 0.4802686256260, 0.2009775476730, 0.0291783426580)
_B1 = ((-2, 9, -18, 11, 0, 0, 0, 0), (0, 1, -6, 3, 2, 0, 0, 0), (0, 0, -2, -3, 6, -1, 0, 0),
       (0, 0, 0, -11, 18, -9, 2, 0), (0, 0, 0, 0, -26, 57, -42, 11))
_B2 = ((-6, 24, -30, 12, 0, 0, 0, 0), (0, 0, 6, -12, 6, 0, 0, 0), (0, 0, 0, 6, -12, 6, 0, 0),
       (0, 0, 0, 12, -30, 24, -6, 0), (0, 0, 0, 0, 18, -48, 42, -12))
_Q = ((-3, 13, -23, 25, 0, 0, 0, 0), (0, 1, -5, 13, 3, 0, 0, 0), (0, 0, -1, 7, 7, -1, 0, 0),
      (0, 0, 0, 3, 13, -5, 1, 0), (0, 0, 0, 0, 25, -23, 13, -3))


def _lin(t, cs):
    acc = None
    for x, k in zip(t, cs):
        if k:
            acc = k * x if acc is None else acc + k * x
    return acc


def _weno7(t):
    """Face value above t[3] from the eight points t[0..7]."""
    beta = []
    for k in range(5):
        third = [0] * k + [-6, 18, -18, 6] + [0] * (4 - k)
        beta.append(2.592e-6 + 720 * _lin(t, _B1[k]) ** 2 + 780 * _lin(t, _B2[k]) ** 2 +
                    781 * _lin(t, third) ** 2)
    top = beta[4]
    for k in range(4):
        top = torch.maximum(top, beta[k])
    beta[4] = top
    wts = [_D[k] / beta[k] for k in range(5)]
    num = sum(wts[k] * _lin(t, _Q[k]) for k in range(5))
    return num / (12 * sum(wts))


def _w5(s, forms):
    """Weighted mean of the candidate values `forms` (value, indicator, factor of the weight)
    on the points s[0..4]; weights 1 / (12e-6 + S)^2 unless given."""
    num = den = 0.0
    for q, wt in forms:
        num, den = num + wt * q, den + wt
    return num / (6.0 * den)


def _closures(P, M, n, lo, hi, ydir, fp, fm):
    """The boundary closures of a CLOSURE direction, in place on the face values P and M
    (faces 0..n along the last axis); fp, fm: the split fluxes with four ghosts."""
    at = lambda a, i: a[..., i + 4]                                       # noqa: E731

    def ind(t0, t1):
        return 13 * t0 * t0 + 3 * t1 * t1

    def stencil(a, i):
        s = [at(a, i + k) for k in range(5)]
        low = ind(s[2] - 2 * s[3] + s[4], 3 * s[2] - 4 * s[3] + s[4])
        mid = ind(s[1] - 2 * s[2] + s[3], s[1] - s[3])
        high = ind(s[0] - 2 * s[1] + s[2], s[0] - 4 * s[1] + 3 * s[2])
        return s, low, mid, high

    def wt(S):
        return 1.0 / (12e-6 + S) ** 2

    def p_forms(i, which):
        s, low, mid, _ = stencil(fp, i)
        q = {"lo": 2 * s[2] + 5 * s[3] - s[4], "mid": -s[1] + 5 * s[2] + 2 * s[3],
             "hi": 2 * s[0] - 7 * s[1] + 11 * s[2]}
        if which == "all":     # products of the other two squares; an indicator not yet summed is 0
            z, a, b = 12e-6 ** 2, (12e-6 + low) ** 2, (12e-6 + mid) ** 2
            return _w5(s, [(q["lo"], z * z), (q["mid"], a * z), (q["hi"], a * b)])
        S = {"lo": low, "mid": mid, "hi": stencil(fp, i)[3]}
        return _w5(s, [(q[k], wt(S[k])) for k in which])

    def m_forms(i, which):
        s = [at(fm, i + k) for k in range(5)]
        S = {"lo": ind(s[4] - 2 * s[3] + s[2], s[4] - 4 * s[3] + 3 * s[2]),
             "mid": ind(s[3] - 2 * s[2] + s[1], s[3] - s[1]),
             "hi": ind(s[2] - 2 * s[1] + s[0], 3 * s[2] - 4 * s[1] + s[0])}
        q = {"lo": 2 * s[4] - 7 * s[3] + 11 * s[2], "mid": -s[3] + 5 * s[2] + 2 * s[1],
             "hi": 2 * s[2] + 5 * s[1] - s[0]}
        return _w5(s, [(q[k], wt(S[k])) for k in which])

    every = ("lo", "mid", "hi")
    if lo:
        P[..., 0] = at(fp, 0)
        P[..., 1] = p_forms(-2, ("lo",))
        P[..., 2] = p_forms(-1, ("lo", "mid"))
        P[..., 3] = p_forms(0, "all")
        M[..., 0] = m_forms(-2, ("lo",))
        M[..., 1] = m_forms(-1, ("mid", "lo"))
        M[..., 2], M[..., 3] = m_forms(0, every), m_forms(1, every)
    if hi:
        P[..., n - 2] = p_forms(n - 5, "all")
        P[..., n - 1] = p_forms(n - 4, ("mid", "hi"))
        M[..., n - 3] = m_forms(n - 5, every)
        M[..., n - 2] = m_forms(n - 4, ("hi", "mid"))
        p1, p2, m1, m2 = at(fp, n - 1), at(fp, n - 2), at(fm, n - 1), at(fm, n - 2)
        if ydir:       # minmod of a difference with itself is the difference
            P[..., n] = p1 + 0.5 * (p1 - p2)
            M[..., n - 1] = m1 - 0.5 * (m1 - m2)
            M[..., n] = M[..., n - 1]      # the last cell's difference of M is left out
        else:
            P[..., n] = 1.5 * p1 - 0.5 * p2
            M[..., n - 1] = M[..., n] = 0.5 * m1 + 0.5 * m2


def _rhs(g, prims, metrics=None, met=None):
    """du of interior primitives (d, u, v, w, T) by the inviscid scheme."""
    du = 0.0
    for axis in range(3):
        dim, n, h = 2 - axis, (g.nx, g.ny, g.nz)[axis], (g.hx, g.hy, g.hz)[axis]
        ext = [_extend(p, g.faces, axis) for p in prims]
        if met is None:
            a, jac = [1.0 if k == axis else 0.0 for k in range(3)], 1.0
            a = [torch.tensor(v, dtype=torch.float64, device=prims[0].device) for v in a]
        else:
            cut = [slice(4, 4 + m) for m in (g.nz, g.ny, g.nx)]
            wide = list(cut)
            wide[dim] = slice(None)
            a, jac = [met[3 * axis + k][tuple(wide)] for k in range(3)], met[9][tuple(cut)]
        fp, fm = (f.movedim(dim + 1, -1) for f in _split(ext[:4], ext[4].sqrt(), a))
        P = _weno7([fp[..., k:k + n + 1] for k in range(8)])
        M = _weno7([fm[..., 7 - k:7 - k + n + 1] for k in range(8)])
        lo, hi = (g.faces[2 * axis + s] == ws.FACE_CLOSURE for s in (0, 1))
        _closures(P, M, n, lo, hi, axis == 1, fp, fm)
        face = (P + M).movedim(-1, dim + 1)
        du = du - jac * (face.narrow(dim + 1, 1, n) - face.narrow(dim + 1, 0, n)) / h
    return du


def _viscous(g, prims, scheme):
    """Viscous terms of du[1..4] on a Cartesian grid."""
    cs = (45 / 60, -9 / 60, 1 / 60) if scheme == 6 else (672 / 840, -168 / 840, 32 / 840, -3 / 840)
    h = (g.hx, g.hy, g.hz)

    def ddx(p, axis):
        dim = p.dim() - 1 - axis
        e, n = _extend(p, g.faces, axis), p.shape[dim]
        return sum(k * (e.narrow(dim, 5 + m, n) - e.narrow(dim, 3 - m, n))
                   for m, k in enumerate(cs)) / h[axis]
    u = prims[1:4]
    T = prims[4]
    gr = [[ddx(p, axis) for axis in range(3)] for p in u]
    div = gr[0][0] + gr[1][1] + gr[2][2]
    tsb = 110.4 / VIS["ref_t"]
    mu = (1.0 + tsb) / VIS["re"] * T ** 1.5 / (tsb + T)
    heat = mu / ((GAMMA - 1.0) * VIS["pr"])
    out = 0.0
    for a in range(3):
        tau = [mu * (gr[a][b] + gr[b][a] - (2.0 / 3.0 * div if a == b else 0.0)) for b in range(3)]
        energy = sum(u[b] * tau[b] for b in range(3)) + heat * ddx(T, a)
        out = out + ddx(torch.stack(tau + [energy]), a)
    return out


def _prims(f):
    d, u, v, w = f[0], f[1] / f[0], f[2] / f[0], f[3] / f[0]
    cv = 1.0 / (GAMMA * (GAMMA - 1.0))
    return [d, u, v, w, (f[4] - 0.5 * d * (u * u + v * v + w * w)) / (d * cv)]


def _step(g, f, dt, viscous=0):
    fn = f
    for krk in (1, 2, 3):
        p = _prims(f)
        du = _rhs(g, p)
        if viscous:
            du[1:] += _viscous(g, p, viscous)
        f = f + dt * du
        if krk > 1:
            f = (3 * fn + f) / 4 if krk == 2 else (fn + 2 * f) / 3
    return f


def exact(c, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "batch":
        if c["grids"] * c["steps"] > 300:
            return None        # a minute of small torch operations
        out = []
        for s in _grids(c, seed):
            g = _grid(c, *s[:3])
            p = _state(*s[:3], c["flow"], s[3], dev)
            f, dt = _cons(p), 0.4 / _max_speed(g, p)
            for _ in range(c["steps"]):
                f = _step(g, f, dt)
            out.append(f.cpu().numpy())
        return out
    g = _grid(c)
    p = _state(g.nx, g.ny, g.nz, c["flow"], seed, dev)
    if c["kind"] == "rhs":
        return _rhs(g, p, met=_metric_fields(g, seed, dev) if c["metrics"] else None)
    f, dt = _cons(p), 0.4 / _max_speed(g, p)
    for _ in range(c["steps"]):
        f = _step(g, f, dt, c["viscous"])
    return f
