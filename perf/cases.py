"""Performance cases of the solver: the work its users have it do, through the
public entry points (FRSolver and the C-ABI), from the 20 x 20 vortex, where
launch latency counts, to the 512 x 512 P5 Taylor-Green run.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) mesh, solver handle and device arrays a program holds
    run(state)          one pass
    work(case)          bytes and flops a pass cannot do without
    exact(case, seed)   what run() returns, in float64 torch, from the scheme's
                        definition (no code of the library)

Operations (`op`):
    step     load a state held on the device, advance n SSP-RK3 steps, read the
             state back on the device: the solver inside a larger program, and
             the benchmark's unit of work
    loop     the driver program's loop: the CFL step once, single advances that
             each wait for the device, the residual norm every tenth step
    gn       one Gauss-Newton product: J V (with the residual), then J^T (J V)
    adjoint  the checkpointed discrete adjoint of n steps
All handles of the process share one compute stream.
"""
import math

import numpy as np
import torch

from zhijian_b200 import _lib as L
from zhijian_b200.meshgen import MixedMesh, QuadMesh
from zhijian_b200.solver import FRSolver, make_params

GAMMA = 1.4
MACH = 0.3
PR = 0.72

# ------------------------------------------------------------------- cases --


def _case(op="step", flow="tgv", nx=64, ny=64, order=3, precision="fp64", scheme="ns", riemann="Roe",
          flux="HU", steps=6, every=0, cfl=0.3):
    """scheme: ns / euler (physics mode), compat (the reference's residual
    semantics, the default of its configuration files).  every: checkpoint
    interval of the adjoint.  cfl: step size over the convective limit; a
    pass costs the same at every step size, and the precision form's runs take
    small ones (a start-up transient), at which FP32 rounding of the residual
    moves the FP64 state by less than 1e-9."""
    return dict(op=op, flow=flow, nx=nx, ny=ny, order=order, precision=precision, scheme=scheme,
                riemann=riemann, flux=flux, steps=steps, every=every, cfl=cfl)


def listed():
    def named(name, **kw):
        return dict(_case(**kw), name=name)
    return [
        # the isentropic vortex of the validation runs, driven step by step
        # from the driver program: launches, synchronisations, host calls
        named("loop-vortex20-p3-euler64", op="loop", flow="vortex", nx=20, ny=20, scheme="euler",
              riemann="Rusanov", steps=20, cfl=0.5),
        # a coarse Navier-Stokes mesh advanced in blocks (parameter studies)
        named("step-tgv20-p3-ns32", nx=20, ny=20, precision="mixed", steps=12, cfl=0.005),
        # a mid-size mesh: about one wave of blocks on the GPU
        named("step-tgv64-p3-ns64", nx=64, ny=64, steps=8),
        # the benchmark mesh: FP64, the precision form, and the reference's
        # semantics in SI units
        named("step-tgv256-p3-ns64", nx=256, ny=256),
        named("step-tgv256-p3-ns32", nx=256, ny=256, precision="mixed", cfl=0.005),
        named("step-si256-p3-compat", flow="si", nx=256, ny=256, scheme="compat", riemann="Rusanov", cfl=0.02),
        # the largest: high order on a fine mesh in the precision form
        named("step-tgv512-p5-ns32", nx=512, ny=512, order=5, precision="mixed", steps=2, cfl=0.005),
        # quads and triangles: the shear layer, precision form at full size
        # and FP64 at an odd size and low order
        named("step-shear384-p3-ns32", flow="shear", nx=384, ny=384, precision="mixed", riemann="HLLC",
              flux="GA", steps=4, cfl=0.005),
        named("step-shear173x141-p2-ns64", flow="shear", nx=173, ny=141, order=2, riemann="HLLC",
              flux="SD", cfl=0.1),
        # curved (Q2) elements at an odd size, inviscid, P4
        named("step-curved149x113-p4-euler64", flow="curved", nx=149, ny=113, order=4, scheme="euler",
              riemann="HLLC", flux="DG"),
        # differentiation: the discrete adjoint's mesh, and a Gauss-Newton
        # product on a ragged one
        named("adjoint-tgv128-p3-ns64", op="adjoint", nx=128, ny=128, steps=8, every=4),
        named("gn-tgv91x57-p2-ns64", op="gn", nx=91, ny=57, order=2),
    ]


# Rough time of one residual per solution point in ns, to keep drawn cases
# below the largest listed one.
_COST = {("ns", "fp64"): 0.14, ("ns", "mixed"): 0.08, ("euler", "fp64"): 0.08, ("euler", "mixed"): 0.05,
         ("compat", "fp64"): 0.055}


def _cost(c):
    t = _COST[(c["scheme"], c["precision"])] * c["nx"] * c["ny"] * (c["order"] + 1) ** 2
    if c["flow"] in ("shear", "curved"):
        t *= 1.5
    if c["op"] == "gn":
        return 8.0 * t
    return 3.0 * c["steps"] * t * (4.0 if c["op"] == "adjoint" else 1.0)


def draw(rng):
    most = 0.9 * max(_cost(c) for c in listed())
    while True:
        op = rng.choices(["step", "loop", "gn", "adjoint"], [7, 1, 1, 1])[0]
        flow = rng.choices(["tgv", "vortex", "shear", "curved", "si"], [5, 1, 2, 1, 1])[0]
        if op in ("gn", "adjoint"):
            flow = "tgv"
        scheme = "compat" if flow == "si" else "ns" if flow == "shear" else rng.choices(["ns", "euler"], [3, 1])[0]
        precision = "fp64" if scheme == "compat" or op in ("gn", "adjoint") else rng.choice(["fp64", "mixed"])
        n = math.exp(rng.uniform(math.log(10.0), math.log(512.0)))
        a = math.exp(rng.uniform(-0.3, 0.3))
        order = rng.choice([1, 2, 3, 3, 4, 5])
        if flow == "curved":
            order = max(2, order)      # a curved Q2 mesh keeps a free stream from P2 on
        if flow == "shear":
            order = min(4, max(2, order))
        c = _case(op=op, flow=flow, nx=max(4, round(n * a)), ny=max(4, round(n / a)), order=order,
                  precision=precision, scheme=scheme,
                  riemann="Rusanov" if scheme == "compat" else rng.choice(["Rusanov", "Roe", "HLLC"]),
                  flux=rng.choice(["DG", "SD", "HU", "GA"]),
                  steps=rng.choice([1, 2, 3, 6, 8, 13]) if op == "step" else rng.choice([4, 6, 8]),
                  every=rng.choice([2, 4, 8]) if op == "adjoint" else 0,
                  cfl=0.005 if precision == "mixed" else 0.02 if scheme == "compat" else
                  0.05 if flow == "shear" else rng.choice([0.1, 0.2, 0.3]))
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------ meshes --

_BOX = {"tgv": (0.0, math.pi), "si": (0.0, math.pi), "curved": (0.0, math.pi), "vortex": (-10.0, 10.0),
        "shear": (0.0, 1.0)}
# boundary names (bottom, right, top, left)
_SIDES = {"tgv": ("slipwall",) * 4, "si": ("slipwall",) * 4, "curved": ("slipwall",) * 4,
          "vortex": ("farfield",) * 4, "shear": ("slipwall", "farfield", "slipwall", "farfield")}
# lattice positions of the nine nodes of a Q2 quadrilateral
_Q2 = [(0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1)]


class _Mesh:
    """Nodes, quadrilaterals [nq, 4 or 9] and triangles [nt, 3] with their
    element numbers, boundary edges (v0, v1, tag); tag 1 + side."""

    def __init__(self, case, seed):
        nx, ny, flow = case["nx"], case["ny"], case["flow"]
        rng = np.random.default_rng([seed, 1])
        q = 2 if flow == "curved" else 1
        lo, hi = _BOX[flow]
        mx, my = q * nx, q * ny
        jj, ii = np.meshgrid(np.arange(my + 1), np.arange(mx + 1), indexing="ij")
        s, t = ii / mx, jj / my
        x, y = lo + (hi - lo) * s, lo + (hi - lo) * t
        if flow in ("tgv", "si"):
            inside = (ii > 0) & (ii < mx) & (jj > 0) & (jj < my)
            x = x + inside * rng.uniform(-0.15, 0.15, x.shape) * (hi - lo) / nx
            y = y + inside * rng.uniform(-0.15, 0.15, y.shape) * (hi - lo) / ny
        if flow == "curved":
            amp = 0.03 * rng.uniform(0.8, 1.0) * (hi - lo)
            x, y = (x + amp * np.sin(np.pi * s) * np.sin(2 * np.pi * t),
                    y + amp * np.sin(2 * np.pi * s) * np.sin(np.pi * t))
        self.xy = np.stack([x.ravel(), y.ravel()], axis=1)
        node = lambda a, b: b * (mx + 1) + a  # noqa: E731
        ej, ei = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
        ei, ej = q * ei.ravel(), q * ej.ravel()
        lat = _Q2 if q == 2 else [(0, 0), (1, 0), (1, 1), (0, 1)]
        quads = np.stack([node(ei + a, ej + b) for a, b in lat], axis=1).astype(np.int64)
        i, j = q * np.arange(nx), q * np.arange(ny)
        sides = [(node(i, 0), node(i + q, 0)), (node(mx, j), node(mx, j + q)),
                 (node(i + q, my), node(i, my)), (node(0, j + q), node(0, j))]
        tag = {n: k + 1 for k, n in enumerate(dict.fromkeys(_SIDES[flow]))}
        self.tag_names = {k: n for n, k in tag.items()}
        self.bnd = np.concatenate([np.stack([a + 0 * b, b + 0 * a, np.full(max(a.size, b.size), tag[n])], axis=1)
                                   for (a, b), n in zip(sides, _SIDES[flow])]).astype(np.int64)
        self.q = q
        if flow == "shear":
            # 30% of the quads, split along a random diagonal
            split = rng.permutation(len(quads)) < round(0.3 * len(quads))
            diag = rng.random(len(quads)) < 0.5
            v = quads.T
            tri = np.where(diag[:, None], np.stack([v[0], v[1], v[2], v[0], v[2], v[3]], axis=1),
                           np.stack([v[0], v[1], v[3], v[1], v[2], v[3]], axis=1))
            first = np.concatenate([[0], np.cumsum(1 + split)])
            self.ids_q, self.quads = first[:-1][~split], quads[~split]
            self.ids_t = np.stack([first[:-1][split], first[:-1][split] + 1], axis=1).ravel()
            self.tris = tri[split].reshape(-1, 3)
            self.n_elem = int(first[-1])
        else:
            self.ids_q, self.quads, self.n_elem = np.arange(len(quads)), quads, len(quads)
            self.ids_t, self.tris = np.zeros(0, np.int64), np.zeros((0, 3), np.int64)

    def of_library(self):
        if len(self.tris) == 0:
            return QuadMesh(self.xy, self.quads, self.bnd, dict(self.tag_names))
        kind = np.ones(self.n_elem, np.int32)
        kind[self.ids_t] = 0
        off = np.concatenate([[0], np.cumsum(3 + kind)]).astype(np.int64)
        conn = np.empty(off[-1], np.int64)
        conn[off[self.ids_q][:, None] + np.arange(4)] = self.quads
        conn[off[self.ids_t][:, None] + np.arange(3)] = self.tris
        return MixedMesh(self.xy, kind, off, conn, self.bnd, dict(self.tag_names))


# ------------------------------------------------------------------ states --

_SI = (1.2, 1.0e5)     # density and pressure of the SI-unit flow


def _state(case, seed, xy):
    """Conserved variables at points xy [..., 2]: the flow with seeded smooth
    perturbations (a few per cent, long waves)."""
    flow = case["flow"]
    rng = np.random.default_rng([seed, 2])
    lo, hi = _BOX[flow]
    x, y = xy[..., 0], xy[..., 1]
    s, t = (x - lo) / (hi - lo), (y - lo) / (hi - lo)

    def wave(amp):
        out = 0.0
        for _ in range(2):
            a, p = rng.uniform(0.5, 1.0) * amp / 2, rng.uniform(0.0, 2 * math.pi, 2)
            k = rng.integers(1, 4, 2)
            out = out + a * torch.sin(math.pi * int(k[0]) * s + p[0]) * torch.sin(math.pi * int(k[1]) * t + p[1])
        return out

    if flow == "vortex":
        f = 5.0 / (2.0 * math.pi) * torch.exp(0.5 * (1.0 - x * x - y * y))
        temp = 1.0 - (GAMMA - 1.0) * f * f / (2.0 * GAMMA)
        rho = temp ** (1.0 / (GAMMA - 1.0))
        u, v, p = 0.5 - f * y, f * x, rho ** GAMMA / GAMMA
    elif flow == "shear":
        rho = torch.ones_like(x)
        u, v = 0.5 * torch.tanh((y - 0.5) / 0.02), 0.01 * torch.sin(2 * math.pi * x)
        p = torch.full_like(x, 1.0 / (GAMMA * MACH * MACH))
    else:
        rho = torch.ones_like(x)
        u, v = torch.sin(x) * torch.cos(y), -torch.cos(x) * torch.sin(y)
        p = 1.0 / (GAMMA * MACH * MACH) + 0.25 * (torch.cos(2 * x) + torch.cos(2 * y))
    rho, p = rho * (1.0 + wave(0.02)), p * (1.0 + wave(0.02))
    u, v = u + wave(0.03), v + wave(0.03)
    if flow == "si":
        scale = _SI[1] / _SI[0] * GAMMA * MACH * MACH       # velocity scale squared
        rho, p = rho * _SI[0], p * _SI[0] * scale
        u, v = u * math.sqrt(scale), v * math.sqrt(scale)
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], dim=-1)


def _free_stream(case):
    """rho, p, Mach number of the far field."""
    if case["flow"] == "si":
        return _SI[0], _SI[1], MACH
    if case["flow"] == "vortex":
        return 1.0, 1.0 / GAMMA, 0.5
    return 1.0, 1.0 / (GAMMA * MACH * MACH), 0.0 if case["flow"] == "shear" else MACH


def _reynolds(case):
    return 2000.0 if case["flow"] == "shear" else 5000.0


def _dt(case):
    lo, hi = _BOX[case["flow"]]
    rho, p, _ = _free_stream(case)
    c = math.sqrt(GAMMA * p / rho)
    speed = c + (1.0 if case["flow"] == "vortex" else MACH * c)     # of the flow's fastest point
    return case["cfl"] * (hi - lo) / max(case["nx"], case["ny"]) / (speed * (2 * case["order"] + 1))


def _direction(seed, shape, device):
    """A seeded random vector of the state's shape."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=device, dtype=torch.float64)


# --------------------------------------------------------------- the passes --

_stream = None


def _compute_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case, st.lib = case, L.lib()
    mesh = _Mesh(case, seed)
    rho, p, mach = _free_stream(case)
    params = make_params(poly_order=case["order"], gamma=GAMMA, rho_inf=rho, p_inf=p, Mach=mach, CFL=case["cfl"],
                         flux_type=case["flux"], riemann=case["riemann"], compat=case["scheme"] == "compat",
                         viscous=case["scheme"] == "ns", Re=_reynolds(case), Pr=PR, precision=case["precision"],
                         bcs=sorted(mesh.tag_names.items()))
    st.solver = s = FRSolver(mesh.of_library(), params)
    st.stream = _compute_stream()
    s.set_stream(st.stream.cuda_stream)
    st.U = _state(case, seed, torch.from_numpy(s.solution_point_coords()).cuda())
    if len(mesh.tris):
        st.U *= torch.from_numpy(s.slot_mask()).cuda()[..., None]
    st.U = st.U.contiguous()
    st.out = torch.empty_like(st.U)
    st.dt = _dt(case)
    if case["op"] in ("gn", "adjoint"):
        st.V = _direction(seed, st.U.shape, "cuda")
    if case["op"] == "gn":
        st.R, st.W = torch.empty_like(st.U), torch.empty_like(st.U)
    torch.cuda.synchronize()
    return st


def run(st):
    s, case = st.solver, st.case
    if case["op"] == "gn":
        s.rhs_jvp(st.U.data_ptr(), st.V.data_ptr(), st.W.data_ptr(), R_ptr=st.R.data_ptr())
        s.rhs_vjp(st.U.data_ptr(), st.W.data_ptr(), st.out.data_ptr())
        return {"R": st.R, "JV": st.W, "JTJV": st.out}
    L.check(st.lib.zj_set_state_device(s.h, st.U.data_ptr()), s.h)
    if case["op"] == "adjoint":
        with torch.cuda.stream(st.stream):
            st.out.copy_(st.V)
        got = s.adjoint_run(st.dt, case["steps"], case["every"], st.out.data_ptr())
        return {"G": st.out, "dRe": got["dRe"]}
    if case["op"] == "loop":
        dt, norms = s.computeTimeStep(), []
        for it in range(case["steps"]):
            s.advance(dt)
            if it % 10 == 0 or it == case["steps"] - 1:
                norms.append(s.computeResidual())
        L.check(st.lib.zj_get_state_device(s.h, st.out.data_ptr()), s.h)
        if case["precision"] == "mixed":     # the norm of an FP32 residual
            norms = [np.float32(n) for n in norms]
        return {"U": st.out, "dt": dt, "norms": norms}
    s.advance(st.dt, case["steps"], sync=False)
    L.check(st.lib.zj_get_state_device(s.h, st.out.data_ptr()), s.h)
    return {"U": st.out}


def work(case):
    """Per residual evaluation: the stage state read and the new one written,
    the base state where the stage uses it (two of three), and per element its
    corners and neighbours; per solution and flux point the arithmetic of the
    sum-factorised scheme.  A Jacobian product counts two residuals, a
    transposed one three."""
    n1 = case["order"] + 1
    elems = case["nx"] * case["ny"] * (1.3 if case["flow"] == "shear" else 1.0)
    per = (0.7 * n1 * n1 + 0.6 * n1 * (n1 + 1) / 2) / 1.3 if case["flow"] == "shear" else n1 * n1
    pts, fps, visc = elems * per, elems * 4.0 * n1, case["scheme"] == "ns"
    flops = (pts * (4 * 4 * n1 * (2 if visc else 1) + 60 + (110 if visc else 0)) +
             fps * (4 * 2 * n1 * (4 if visc else 2) + 110 + (100 if visc else 0)))
    geom = elems * (4 * 16 + 4 * 8)
    if case["op"] == "gn":
        return {"bytes": pts * 32 * 6 + 2 * geom, "flops": 5 * flops}
    stage = pts * (64 + 32 * 2 / 3) + geom
    n = 3 * case["steps"]
    if case["op"] == "adjoint":
        return {"bytes": n * stage + n * (pts * 32 * 3 + geom), "flops": 4 * n * flops}
    return {"bytes": n * stage, "flops": n * flops}


# --------------------------------------------------- the scheme, in float64 --

def _lagrange(nodes, x):
    """Values and derivatives [len(x), n] of the Lagrange polynomials."""
    n = len(nodes)
    val, der = np.ones((len(x), n)), np.zeros((len(x), n))
    for j in range(n):
        for m in range(n):
            if m != j:
                val[:, j] *= (x - nodes[m]) / (nodes[j] - nodes[m])
        for k in range(n):
            if k == j:
                continue
            term = np.full(len(x), 1.0 / (nodes[j] - nodes[k]))
            for m in range(n):
                if m not in (j, k):
                    term *= (x - nodes[m]) / (nodes[j] - nodes[m])
            der[:, j] += term
    return val, der


def _legendre_der(n, x):
    return np.polynomial.legendre.Legendre.basis(n).deriv()(x)


def _vcjh_c(p, flux):
    ap2 = (math.factorial(2 * p) / (2.0 ** p * math.factorial(p))) ** 2
    return {"DG": 0.0, "SD": 2.0 * p / ((2.0 * p + 1.0) * (p + 1.0) * ap2),
            "HU": 2.0 * (p + 1.0) / ((2.0 * p + 1.0) * p * ap2),
            "GA": 2.0 * (p + 1.0) * math.factorial(p) ** 2 / (math.factorial(2 * p) * (2.0 * p + 1.0))}[flux]


class _Quad:
    """Dense operators of a quadrilateral: Dr, Ds [n, n], L [4 n1, n] (edge
    interpolation), Phi [n, 4 n1] (divergence of the correction fields)."""
    nref = np.array([[0.0, -1.0], [1.0, 0.0], [0.0, 1.0], [-1.0, 0.0]])

    def __init__(self, p, flux, compat):
        n1 = p + 1
        g = np.polynomial.legendre.leggauss(n1)[0]
        one = np.eye(n1)
        d = _lagrange(g, g)[1]
        self.Dr, self.Ds = np.kron(one, d), np.kron(d, one)
        self.r, self.s = np.tile(g, n1), np.repeat(g, n1)
        f = np.ones(n1)
        self.fr, self.fs = np.concatenate([g, f, -g, -f]), np.concatenate([-f, g, f, -g])
        self.L = np.einsum("qi,qj->qji", _lagrange(g, self.fr)[0], _lagrange(g, self.fs)[0]).reshape(4 * n1, n1 * n1)
        ap2 = (math.factorial(2 * p) / (2.0 ** p * math.factorial(p))) ** 2
        eta = _vcjh_c(p, flux) * (2 * p + 1) * ap2 / 2.0
        if compat:
            eta = 0.0          # the Radau correction, whatever the flux type

        def right(x):
            return 0.5 * (_legendre_der(p, x) + (eta * _legendre_der(p - 1, x) + _legendre_der(p + 1, x)) / (1.0 + eta))
        gR, gL = right(g), -right(-g)
        rev = one[::-1]
        if compat:     # the reference's signs, and edges 2, 3 in unreversed order
            blocks = [np.kron(gL[:, None], one), np.kron(one, gR[:, None]), np.kron(gR[:, None], one),
                      np.kron(one, gL[:, None])]
        else:
            blocks = [-np.kron(gL[:, None], one), np.kron(one, gR[:, None]), np.kron(gR[:, None], rev),
                      -np.kron(rev, gL[:, None])]
        self.Phi = np.concatenate(blocks, axis=1)

    def shape(self, q, r, s):
        """Derivatives of the element map's node functions in the mesh's node order."""
        nodes = np.linspace(-1.0, 1.0, q + 1)
        (vr, dr), (vs, ds) = _lagrange(nodes, r), _lagrange(nodes, s)
        lat = _Q2 if q == 2 else [(0, 0), (1, 0), (1, 1), (0, 1)]
        return (np.stack([dr[:, a] * vs[:, b] for a, b in lat], axis=1),
                np.stack([vr[:, a] * ds[:, b] for a, b in lat], axis=1))


class _Tri:
    """The same for a triangle, from a monomial basis; the correction fields
    solve (M + c K) phi = b (Castonguay, Vincent & Jameson 2012)."""
    nref = np.array([[0.0, -1.0], [math.sqrt(0.5), math.sqrt(0.5)], [-1.0, 0.0]])

    def __init__(self, p, flux):
        n1 = p + 1
        mono = [(a, b) for a in range(n1) for b in range(n1 - a)]
        g, w = np.polynomial.legendre.leggauss(n1)
        pts = [(0.5 * (1 + g[i]), 0.5 * (1 + g[j])) for j in range(n1) for i in range(n1 - j)]
        self.r = np.array([2 * a * (1 - b) - 1 for a, b in pts])
        self.s = np.array([2 * b - 1 for a, b in pts])
        val = lambda r, s: np.stack([r ** a * s ** b for a, b in mono], axis=-1)  # noqa: E731
        inv = np.linalg.inv(val(self.r, self.s))
        self.Dr = np.stack([a * self.r ** max(a - 1, 0) * self.s ** b for a, b in mono], axis=-1) @ inv
        self.Ds = np.stack([b * self.r ** a * self.s ** max(b - 1, 0) for a, b in mono], axis=-1) @ inv
        f = np.ones(n1)
        self.fr, self.fs = np.concatenate([g, -g, -f]), np.concatenate([-f, g, -g])
        edge = val(self.fr, self.fs)
        self.L = edge @ inv
        xq, wq = np.polynomial.legendre.leggauss(2 * p + 3)
        a, b = np.meshgrid(xq, xq, indexing="ij")
        wt = (np.outer(wq, wq) * 0.5 * (1 - b)).ravel()
        mq = val((0.5 * (1 + a) * (1 - b) - 1).ravel(), b.ravel())
        mass = (mq * wt[:, None]).T @ mq
        c = _vcjh_c(p, flux)
        for i, (m, n) in enumerate(mono):
            if m + n == p:
                mass[i, i] += c * math.comb(p, m) * (math.factorial(m) * math.factorial(n)) ** 2 * 2.0
        half = np.repeat([1.0, math.sqrt(2.0), 1.0], n1) * np.tile(w, 3)
        self.Phi = val(self.r, self.s) @ np.linalg.solve(mass, (half[:, None] * edge).T)

    def shape(self, q, r, s):
        one = np.ones_like(r)
        return (np.stack([-0.5 * one, 0.5 * one, 0 * one], axis=1), np.stack([-0.5 * one, 0 * one, 0.5 * one], axis=1))


class _Scheme:
    """Residual of a case on its mesh, on torch tensors in float64."""

    def __init__(self, case, seed, device):
        self.case, self.device = case, device
        self.compat, self.viscous = case["scheme"] == "compat", case["scheme"] == "ns"
        self.riemann, self.n1 = case["riemann"], case["order"] + 1
        mesh = self.mesh = _Mesh(case, seed)
        self.E, n1 = mesh.n_elem, self.n1
        to = self.to
        kinds = [(_Quad(case["order"], case["flux"], self.compat), mesh.ids_q, mesh.quads, 4)]
        if len(mesh.tris):
            kinds.append((_Tri(case["order"], case["flux"]), mesh.ids_t, mesh.tris, 3))
        # faces: edge rows e*4 + l by their end nodes; the lower row is the left side
        rows, ends = [], []
        for k, ids, conn, nv in kinds:
            for l in range(nv):
                rows.append(ids * 4 + l)
                ends.append(np.sort(np.stack([conn[:, l], conn[:, (l + 1) % nv]], axis=1), axis=1))
        rows, ends = np.concatenate(rows), np.concatenate(ends)
        key = ends[:, 0] * (len(mesh.xy) + 1) + ends[:, 1]
        o = np.lexsort((rows, key))
        rows, key = rows[o], key[o]
        pair = np.nonzero(key[1:] == key[:-1])[0]
        nbr, left = np.full(4 * self.E, -1, np.int64), np.ones(4 * self.E, bool)
        nbr[rows[pair]], nbr[rows[pair + 1]], left[rows[pair + 1]] = rows[pair + 1], rows[pair], False
        tags = {}
        for a, b, t in mesh.bnd:
            tags[min(a, b) * (len(mesh.xy) + 1) + max(a, b)] = mesh.tag_names[int(t)]
        open_rows = nbr[rows] < 0
        wall = np.zeros(4 * self.E, bool)
        for r, k in zip(rows[open_rows], key[open_rows]):
            wall[r] = tags[k] == "slipwall"
        used = np.zeros(4 * self.E, bool)
        used[rows] = True
        self.bnd = to(np.nonzero((nbr < 0) & used)[0])
        self.wall = to(wall)[self.bnd][:, None]
        self.nbr = to(np.where(nbr < 0, 0, nbr))
        self.inner = to(nbr >= 0)[:, None, None]
        self.left = to(left)[:, None]
        # metrics at the solution points; normals and edge scales at the flux points
        nrm = torch.zeros(4 * self.E, n1, 3, dtype=torch.float64, device=device)
        nrm[..., 0] = 1.0
        self.kinds = []
        for k, ids, conn, nv in kinds:
            xy = mesh.xy[conn]
            a, b = k.shape(mesh.q, k.r, k.s)
            xr, xs = np.einsum("na,eac->enc", a, xy), np.einsum("na,eac->enc", b, xy)
            J = xr[..., 0] * xs[..., 1] - xs[..., 0] * xr[..., 1]
            A = np.stack([xs[..., 1], -xs[..., 0], -xr[..., 1], xr[..., 0]], axis=-1)     # J * Jinv
            a, b = k.shape(mesh.q, k.fr, k.fs)
            xr, xs = np.einsum("na,eac->enc", a, xy), np.einsum("na,eac->enc", b, xy)
            nr = np.repeat(k.nref, n1, axis=0)
            tan = xs * nr[:, None, 0].T[..., None] - xr * nr[:, None, 1].T[..., None]
            s = np.hypot(tan[..., 0], tan[..., 1])
            rec = np.stack([tan[..., 1] / s, -tan[..., 0] / s, s], axis=-1).reshape(len(ids), nv, n1, 3)
            for l in range(nv):
                nrm[to(ids * 4 + l)] = to(rec[:, l])
            ops = [to(m) for m in (k.Dr, k.Ds, k.L, k.Phi, nr)]
            self.kinds.append((to(ids), nv, len(k.r), ops, to(J)[..., None], to(A), to(xy)))
        # a right side's normal is the left element's, at the coinciding point;
        # the edge scale is the element's own
        flip = torch.cat([nrm[self.nbr].flip(1)[..., :2], nrm[..., 2:]], -1)
        self.nrm = torch.where(self.left[..., None], nrm, flip)
        self.points = self._points(kinds)

    def to(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.device)

    def _points(self, kinds):
        xy = torch.zeros(self.E, self.n1 ** 2, 2, dtype=torch.float64, device=self.device)
        for (k, ids, conn, nv), (_, _, n, _, _, _, nodes) in zip(kinds, self.kinds):
            if nv == 3:
                w = np.stack([-0.5 * (k.r + k.s), 0.5 * (1 + k.r), 0.5 * (1 + k.s)], axis=1)
            else:
                q = self.mesh.q
                lat = _Q2 if q == 2 else [(0, 0), (1, 0), (1, 1), (0, 1)]
                vr, vs = (_lagrange(np.linspace(-1.0, 1.0, q + 1), z)[0] for z in (k.r, k.s))
                w = np.stack([vr[:, a] * vs[:, b] for a, b in lat], axis=1)
            xy[self.to(ids), :n] = torch.einsum("na,eac->enc", self.to(w), nodes)
        return xy

    def state(self, seed):
        U = _state(self.case, seed, self.points)
        for ids, nv, n, *_ in self.kinds:
            if n < U.shape[1]:
                mask = torch.ones_like(U[:, :, :1])
                mask[ids, n:] = 0.0
                U = U * mask
        return U

    # -- pointwise physics (last axis: variables)
    @staticmethod
    def prim(U):
        u, v = U[..., 1] / U[..., 0], U[..., 2] / U[..., 0]
        return U[..., 0], u, v, (GAMMA - 1.0) * (U[..., 3] - 0.5 * U[..., 0] * (u * u + v * v))

    def flux(self, U):
        r, u, v, p = self.prim(U)
        return (torch.stack([U[..., 1], U[..., 1] * u + p, U[..., 1] * v, (U[..., 3] + p) * u], -1),
                torch.stack([U[..., 2], U[..., 2] * u, U[..., 2] * v + p, (U[..., 3] + p) * v], -1))

    def viscous_flux(self, U, X, Y, Re):
        r, u, v, p = self.prim(U)
        T = p / r
        grad = []
        for D in (X, Y):
            du, dv = (D[..., 1] - u * D[..., 0]) / r, (D[..., 2] - v * D[..., 0]) / r
            dp = (GAMMA - 1.0) * (D[..., 3] - 0.5 * D[..., 0] * (u * u + v * v) - r * (u * du + v * dv))
            grad.append((du, dv, (dp - T * D[..., 0]) / r))
        (ux, vx, tx), (uy, vy, ty) = grad
        mu = T ** 0.7 / Re
        k = mu * GAMMA / ((GAMMA - 1.0) * PR)
        lam = -2.0 / 3.0 * mu * (ux + vy)
        xx, yy, xy = 2 * mu * ux + lam, 2 * mu * vy + lam, mu * (uy + vx)
        z = torch.zeros_like(xx)
        return (torch.stack([z, xx, xy, u * xx + v * xy + k * tx], -1),
                torch.stack([z, xy, yy, u * xy + v * yy + k * ty], -1))

    def common(self, A, B, nx, ny):
        """Riemann flux along n, A on the left."""
        (rA, uA, vA, pA), (rB, uB, vB, pB) = self.prim(A), self.prim(B)
        n = torch.stack([torch.zeros_like(nx), nx, ny, torch.zeros_like(nx)], -1)
        qA, qB = uA * nx + vA * ny, uB * nx + vB * ny
        e3 = torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=torch.float64, device=A.device)
        FA = A * qA[..., None] + pA[..., None] * (n + e3 * qA[..., None])
        FB = B * qB[..., None] + pB[..., None] * (n + e3 * qB[..., None])
        cA, cB = torch.sqrt(GAMMA * pA / rA), torch.sqrt(GAMMA * pB / rB)
        if self.riemann == "Rusanov" or self.compat:
            s = torch.maximum(torch.sqrt(uA * uA + vA * vA) + cA, torch.sqrt(uB * uB + vB * vB) + cB)
            return 0.5 * (FA + FB) - 0.5 * s[..., None] * (B - A)
        if self.riemann == "Roe":
            a, b = torch.sqrt(rA), torch.sqrt(rB)
            mean = lambda x, y: (a * x + b * y) / (a + b)  # noqa: E731
            u, v, H = mean(uA, uB), mean(vA, vB), mean((A[..., 3] + pA) / rA, (B[..., 3] + pB) / rB)
            r, q, qq = a * b, u * nx + v * ny, u * u + v * v
            c = torch.sqrt((GAMMA - 1.0) * (H - 0.5 * qq))
            eps = 0.1 * c
            fix = lambda l: torch.where(l < eps, (l * l + eps * eps) / (2 * eps), l)  # noqa: E731
            l1, l2, l4 = fix((q - c).abs()), q.abs(), fix((q + c).abs())
            dp, dq = pB - pA, (uB - uA) * nx + (vB - vA) * ny
            w1, w4 = l1 * (dp - r * c * dq) / (2 * c * c), l4 * (dp + r * c * dq) / (2 * c * c)
            w2, w3 = l2 * (rB - rA - dp / (c * c)), l2 * r * ((vB - vA) * nx - (uB - uA) * ny)
            d = torch.stack([w1 + w2 + w4,
                             w1 * (u - c * nx) + w2 * u - w3 * ny + w4 * (u + c * nx),
                             w1 * (v - c * ny) + w2 * v + w3 * nx + w4 * (v + c * ny),
                             w1 * (H - c * q) + w2 * 0.5 * qq + w3 * (v * nx - u * ny) + w4 * (H + c * q)], -1)
            return 0.5 * (FA + FB) - 0.5 * d
        ps = (0.5 * (pA + pB) - 0.125 * (qB - qA) * (rA + rB) * (cA + cB)).clamp(min=1e-10)
        k = (GAMMA + 1.0) / (2.0 * GAMMA)
        fan = lambda p: torch.where(ps <= p, torch.ones_like(p), torch.sqrt(1.0 + k * (ps / p - 1.0)))  # noqa: E731
        SA, SB = qA - cA * fan(pA), qB + cB * fan(pB)
        SM = (pB - pA + rA * qA * (SA - qA) - rB * qB * (SB - qB)) / (rA * (SA - qA) - rB * (SB - qB))

        def side(U, F, r, u, v, p, q, S):
            f = r * (S - q) / (S - SM)
            star = torch.stack([f, f * (u + (SM - q) * nx), f * (v + (SM - q) * ny),
                                f * (U[..., 3] / r + (SM - q) * (SM + p / (r * (S - q))))], -1)
            return F + S[..., None] * (star - U)
        F = torch.where((SM >= 0)[..., None], side(A, FA, rA, uA, vA, pA, qA, SA), side(B, FB, rB, uB, vB, pB, qB, SB))
        return torch.where((SA >= 0)[..., None], FA, torch.where((SB <= 0)[..., None], FB, F))

    def ghost(self, U, nx, ny):
        r, u, v, p = self.prim(U)
        q = u * nx + v * ny
        slip = (r, u - 2 * q * nx, v - 2 * q * ny, p)
        ri, pi, mach = _free_stream(self.case)
        ci = math.sqrt(GAMMA * pi / ri)
        ui = mach * ci
        qi = ui * nx
        c = torch.sqrt(GAMMA * p / r)
        up, dn = q + 2 * c / (GAMMA - 1.0), qi - 2 * ci / (GAMMA - 1.0)
        qb, cb = 0.5 * (up + dn), 0.25 * (GAMMA - 1.0) * (up - dn)
        out = qb >= 0
        vt = torch.where(out, v * nx - u * ny, -ui * ny)
        s = torch.where(out, p / r ** GAMMA, torch.full_like(p, pi / ri ** GAMMA))
        rb = (cb * cb / (GAMMA * s)) ** (1.0 / (GAMMA - 1.0))
        far = (rb, qb * nx - vt * ny, qb * ny + vt * nx, rb * cb * cb / GAMMA)
        r, u, v, p = (torch.where(self.wall, a, b) for a, b in zip(slip, far))
        return torch.stack([r, r * u, r * v, p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)], -1)

    # -- element operators
    def traces(self, fields):
        """Edge rows [4 E, n1, m] of per-kind nodal fields [e, n, m]."""
        m = fields[0].shape[-1]
        idx, val = [], []
        for (ids, nv, n, (Dr, Ds, Lq, Phi, nr), *_), f in zip(self.kinds, fields):
            idx.append((ids[:, None] * 4 + torch.arange(nv, device=self.device)).reshape(-1))
            val.append((Lq @ f).reshape(-1, self.n1, m))
        base = torch.ones(4 * self.E, self.n1, m, dtype=torch.float64, device=self.device)
        return base.index_copy(0, torch.cat(idx), torch.cat(val))

    def own(self, rows, ids, nv):
        """Flux points [e, nv n1, m] of elements ids."""
        m = rows.shape[-1]
        return rows.reshape(self.E, 4, self.n1, m)[ids, :nv].reshape(len(ids), nv * self.n1, m)

    def residual(self, U, Re):
        nx, ny, s = self.nrm.unbind(-1)
        Us = [U[ids, :n] for ids, nv, n, *_ in self.kinds]
        T = self.traces(Us)
        other = T[self.nbr].flip(1)
        g = self.ghost(T[self.bnd], nx[self.bnd], ny[self.bnd])
        other = other.index_copy(0, self.bnd, g)
        left = self.left[..., None]
        A, B = torch.where(left, T, other), torch.where(left, other, T)
        Fc = self.common(A, B, nx, ny)
        fluxes = [self.flux(u) for u in Us]
        if self.viscous:
            jump = 0.5 * (other - T)
            Q = []
            for (ids, nv, n, (Dr, Ds, Lq, Phi, nr), J, M, _), u in zip(self.kinds, Us):
                d = self.own(jump, ids, nv)
                dr = Dr @ u + Phi @ (d * nr[:, :1])
                ds = Ds @ u + Phi @ (d * nr[:, 1:])
                Q.append(torch.cat([(M[..., :1] * dr + M[..., 2:3] * ds) / J,
                                    (M[..., 1:2] * dr + M[..., 3:] * ds) / J], -1))
            fluxes = [tuple(f - fv for f, fv in zip(fl, self.viscous_flux(u, q[..., :4], q[..., 4:], Re)))
                      for fl, u, q in zip(fluxes, Us, Q)]
            TQ = self.traces(Q)
            mean = torch.where(self.inner, 0.5 * (TQ + TQ[self.nbr].flip(1)), TQ)
            Fv, Gv = self.viscous_flux(0.5 * (A + B), mean[..., :4], mean[..., 4:], Re)
            Fn = Fv * nx[..., None] + Gv * ny[..., None]
            b, bx, by = Fn[self.bnd], nx[self.bnd], ny[self.bnd]
            tnn, z = b[..., 1] * bx + b[..., 2] * by, torch.zeros_like(bx)
            closed = torch.stack([b[..., 0], tnn * bx, tnn * by, z], -1)
            Fn = Fn.index_copy(0, self.bnd, torch.where(self.wall[..., None], closed, b))
            Fc = Fc - Fn
        sign = torch.where(self.left, 1.0, -1.0).to(torch.float64)
        Fs = (sign * s)[..., None] * Fc
        R = torch.zeros_like(U)
        for (ids, nv, n, (Dr, Ds, Lq, Phi, nr), J, M, _), (F, G) in zip(self.kinds, fluxes):
            Ft, Gt = M[..., :1] * F + M[..., 1:2] * G, M[..., 2:3] * F + M[..., 3:] * G
            dF = self.own(Fs, ids, nv) - ((Lq @ Ft) * nr[:, :1] + (Lq @ Gt) * nr[:, 1:])
            R = R.index_put((ids[:, None], torch.arange(n, device=self.device)[None]),
                            -(Dr @ Ft + Ds @ Gt + Phi @ dF) / J)
        return R

    def residual_compat(self, U):
        """The reference's residual: unscaled corrections, a right side's flux
        difference at the left side's point of the same number."""
        nx, ny, s = self.nrm.unbind(-1)
        ids, nv, n, (Dr, Ds, Lq, Phi, nr), J, M, _ = self.kinds[0]
        T = self.traces([U])
        other = T[self.nbr].flip(1)
        other = other.index_copy(0, self.bnd, self.ghost(T[self.bnd], nx[self.bnd], ny[self.bnd]))
        left = self.left[..., None]
        Fc = self.common(torch.where(left, T, other), torch.where(left, other, T), nx, ny)
        Fc = torch.where(left, Fc, Fc.flip(1))
        F, G = self.flux(T)
        dF = torch.where(left, 1.0, -1.0) * (Fc - F * nx[..., None] - G * ny[..., None])
        F, G = self.flux(U)
        div = (M[..., :1] * (Dr @ F) + M[..., 2:3] * (Ds @ F) + M[..., 1:2] * (Dr @ G) + M[..., 3:] * (Ds @ G)) / J
        return -div - Phi @ self.own(dF, ids, nv)

    @staticmethod
    def clamp(U):
        r = U[..., 0].clamp(0.01, 100.0)
        u, v = U[..., 1] / r, U[..., 2] / r
        m = torch.sqrt(u * u + v * v)
        k = torch.where(m > 2000.0, 2000.0 / m, torch.ones_like(m))
        u, v = u * k, v * k
        ke = 0.5 * r * (u * u + v * v)
        p = (0.4 * (U[..., 3] - ke)).clamp(100.0, 1e8)
        return torch.stack([r, r * u, r * v, p / 0.4 + ke], -1)

    def step(self, U, dt, Re):
        """One SSP-RK3 step: the new state and the last stage's residual."""
        rhs = self.residual_compat if self.compat else lambda X: self.residual(X, Re)
        fix = self.clamp if self.compat else lambda X: X
        A = fix(U + dt * rhs(U))
        B = fix(0.75 * U + 0.25 * A + 0.25 * dt * rhs(A))
        R = rhs(B)
        return fix(U / 3.0 + 2.0 / 3.0 * B + 2.0 / 3.0 * dt * R), R


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    sch = _Scheme(case, seed, device)
    U, Re = sch.state(seed), torch.tensor(_reynolds(case), dtype=torch.float64, device=device)
    if case["op"] == "gn":
        V = _direction(seed, U.shape, device)
        R, JV = torch.func.jvp(lambda X: sch.residual(X, Re), (U,), (V,))
        X = U.clone().requires_grad_()
        W, = torch.autograd.grad(sch.residual(X, Re), X, JV)
        return {"R": R, "JV": JV, "JTJV": W}
    dt = _dt(case)
    if case["op"] == "adjoint":
        G = _direction(seed, U.shape, device)
        states = [U]
        with torch.no_grad():
            for _ in range(case["steps"] - 1):
                states.append(sch.step(states[-1], dt, Re)[0])
        dRe = torch.zeros_like(Re)
        for U in reversed(states):
            X, r = U.clone().requires_grad_(), Re.clone().requires_grad_()
            G, d = torch.autograd.grad(sch.step(X, dt, r)[0], (X, r), G, allow_unused=True)
            dRe = dRe + (d if d is not None else 0.0)
        return {"G": G, "dRe": float(dRe)}
    with torch.no_grad():
        if case["op"] == "step":
            for _ in range(case["steps"]):
                U, _ = sch.step(U, dt, Re)
            return {"U": U}
        # the CFL step over all points, then the driver's loop
        speeds = []
        for ids, nv, n, *_ in sch.kinds:
            r, u, v, p = sch.prim(U[ids, :n])
            xy = torch.from_numpy(sch.mesh.xy[sch.mesh.quads if nv == 4 else sch.mesh.tris][:, :nv]).to(device)
            x, y = xy.unbind(-1)
            area = 0.5 * (x * y.roll(-1, 1) - y * x.roll(-1, 1)).sum(1).abs()
            speeds.append((area.sqrt()[:, None] / (torch.sqrt(u * u + v * v) + torch.sqrt(GAMMA * p / r))).min())
        dt, norms = case["cfl"] * float(min(speeds)) / (2 * case["order"] + 1), []
        for it in range(case["steps"]):
            U, R = sch.step(U, dt, Re)
            if it % 10 == 0 or it == case["steps"] - 1:
                norms.append(float(torch.sqrt((R * R).sum())))
        return {"U": U, "dt": dt, "norms": norms}
