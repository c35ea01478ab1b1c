"""Work that users of the library have it do, as cases that can be timed.

A case is one call sequence through the public Python classes (``Handle``,
``Batch``, ``Mpnn`` of ``cfdsfemmpi_b200``): a time step of one flow problem
from a given state, the same for a batch of independent problems, or the
gradient of the guess network's loss.  A program has its handle (mesh, pattern,
symbolic factorisation, device buffers) for thousands of time steps, so
``prepare`` makes the handle and the state vectors in pinned host memory, and
``run`` hands the state over, takes the step and reads the solution back.

Time steps are solved as far as 64 bits allow (relative tolerance 1e-15 for
BiCGStab, 1e-14 for GMRES and for the true residual in mixed precision).  In an
enclosed cavity the pressure level is held by a single pinned node, so it is
the part of the answer that a solve determines last: at 64 elements per side
and Re 1000 a change of the state in its last bit moves it by 1e-9 of the
answer, at Re 100 by 5e-11.  With these tolerances and Reynolds numbers two
correct solves agree to about ten digits in every field and can be compared.

Fields of a case:
  work     "step", "batch" or "net"
  mesh     "quad" / "tri" (2D cavity), "hex" / "tet" (graded 3D cavity), "wake" (O-grid around a cylinder)
  n, nr    elements per side; on the wake n around and nr outward
  ksp, pc, levels, restart   solver (PETSc's names; levels = -1 with preonly is the direct solve)
  precision, guess           "fp64" or "mixed"; "constant", "extrapolation" or "network"
  re       Reynolds number (unit speed and length)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cfdsfemmpi_b200 import io, meshgen
from cfdsfemmpi_b200._lib import Batch, Handle, Mpnn

HID, LAYERS, FIN, FOUT = 64, 3, 16, 16        # shape of the guess network
NET_PARAMS = FIN * HID + HID + LAYERS * (2 * HID * HID + HID) + HID * FOUT + FOUT
DENSE_LIMIT = 20000                           # largest system that exact() solves densely


def _step(name, mesh, n, ksp, pc, levels=0, restart=30, nr=0, precision="fp64", guess="constant", re=100.0):
    c = {"work": "step", "mesh": mesh, "n": n, "nr": nr, "ksp": ksp, "pc": pc, "levels": levels, "restart": restart,
         "precision": precision, "guess": guess, "re": re}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's 10 x 10 known-answer cavity with GMRES(50) + Jacobi: a few hundred unknowns, where the
        # latency of one small kernel after another is all there is
        _step("quad10_gmres_jacobi", "quad", 10, "gmres", "jacobi", restart=50),
        # one mid-size 2D cavity with an odd side, alone: the restarted GMRES with the point-block preconditioner
        _step("quad57_gmres_pbjacobi", "quad", 57, "gmres", "pbjacobi", restart=400, re=400.0),
        # parameter study: independent cavities of uneven size and Reynolds number stepped together
        {"name": "batch12_quad", "work": "batch", "mesh": "quad", "count": 12, "n": 24, "n_hi": 64, "restart": 400,
         "pc": "pbjacobi"},
        # the reference's tests solve directly (preonly + LU): a complete factorisation each step
        _step("quad64_direct", "quad", 64, "preonly", "bjacobi", levels=-1, re=400.0),
        # vortex street behind a cylinder with the reference's BiCGStab + ILU(3) option file
        _step("wake256_bcgs_ilu3", "wake", 256, "bcgs", "bjacobi", levels=3, nr=128),
        # small and odd 3D cavity: fewer rows than the chip has warps
        _step("hex11_bcgs_ilu0", "hex", 11, "bcgs", "bjacobi"),
        # tetrahedral mesh, GMRES and point-block Jacobi
        _step("tet14_gmres_pbjacobi", "tet", 14, "gmres", "pbjacobi", restart=200),
        # the 3D cavity of the benchmark configurations, ordinary and large, with BiCGStab + ILU(0)
        _step("hex32_bcgs_ilu0", "hex", 32, "bcgs", "bjacobi"),
        _step("hex64_bcgs_ilu0", "hex", 64, "bcgs", "bjacobi"),
        # the same physics in mixed precision, started from the learned and extrapolated guess
        _step("hex32_mixed_network", "hex", 32, "gmres", "bjacobi", precision="mixed", guess="network"),
        # training of the guess network: loss and gradient (forward and backward) of one sample
        {"name": "net_hex32", "work": "net", "mesh": "hex", "n": 32},
        {"name": "net_hex64", "work": "net", "mesh": "hex", "n": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind of work by chance, its size over the logarithm of the range."""
    re = round(10.0 ** rng.uniform(2.0, 2.5), 1)
    kind = rng.choice(["quad_gmres", "quad_direct", "quad_ilu", "wake", "hex", "hex", "mixed", "tet", "batch", "net"])
    if kind == "quad_gmres":
        n = _log_int(rng, 5, 72)
        if n <= 24:
            return _step(None, "quad", n, "gmres", rng.choice(["jacobi", "pbjacobi"]), restart=rng.choice([50, 200]))
        return _step(None, "quad", n, "gmres", "pbjacobi", restart=400, re=re)
    if kind == "quad_direct":
        return _step(None, rng.choice(["quad", "tri"]), _log_int(rng, 6, 64), "preonly", "bjacobi", levels=-1, re=re)
    if kind == "quad_ilu":
        return _step(None, "quad", _log_int(rng, 8, 128), "bcgs", "bjacobi", levels=rng.choice([0, 1, 3]), re=re)
    if kind == "wake":
        n = _log_int(rng, 64, 224)
        return _step(None, "wake", n, "bcgs", "bjacobi", levels=rng.choice([1, 2, 3]), nr=max(24, n // 2 + rng.randint(-7, 7)))
    if kind == "hex":
        n = _log_int(rng, 6, 60)
        return _step(None, "hex", n, "bcgs", "bjacobi", levels=1 if n <= 32 and rng.random() < 0.3 else 0, re=re)
    if kind == "mixed":
        return _step(None, "hex", _log_int(rng, 8, 40), "gmres", "bjacobi", precision="mixed",
                     guess=rng.choice(["constant", "extrapolation", "network"]), re=re)
    if kind == "tet":
        n = _log_int(rng, 4, 20)
        if rng.random() < 0.5:
            return _step(None, "tet", n, "gmres", "pbjacobi", restart=200)
        return _step(None, "tet", n, "bcgs", "bjacobi", re=re)
    if kind == "batch":
        n = rng.randint(12, 32)
        return {"work": "batch", "mesh": "quad", "count": rng.randint(2, 16), "n": n, "n_hi": n + rng.randint(4, 32),
                "restart": 400, "pc": "pbjacobi"}
    mesh = rng.choice(["quad", "hex"])
    return {"work": "net", "mesh": mesh, "n": _log_int(rng, 16, 160) if mesh == "quad" else _log_int(rng, 6, 60)}


# ---------------------------------------------------------------------------
# meshes, controls and states

def _mesh(case, n=None):
    n = case["n"] if n is None else n
    kind = case["mesh"]
    if kind == "wake":
        return meshgen.cylinder_ogrid(n, case["nr"])
    base = meshgen.cavity2d(n) if kind in ("quad", "tri") else meshgen.cavity3d(n)
    split = {"tri": ([0, 1, 2], [0, 2, 3]),
             "tet": ([0, 1, 3, 4], [1, 2, 3, 6], [1, 3, 4, 6], [1, 4, 5, 6], [3, 4, 6, 7])}.get(kind)
    if split is None:
        return base
    conn = np.ascontiguousarray(np.concatenate([base.conn[:, s] for s in split]).astype(np.int32))
    return io.Mesh(ndim=base.ndim, npElem=conn.shape[1], coords=base.coords, conn=conn, dbc=base.dbc,
                   output_nodes=base.output_nodes)


def _modes(X, rng, amplitude):
    """A smooth velocity that vanishes on the walls of the unit square / cube (curl of a few modes) and a smooth
    pressure that vanishes at the origin: what a developing cavity flow looks like."""
    nd = X.shape[1]
    f = np.zeros((X.shape[0], nd + 1))
    s2 = lambda x, k: np.sin(math.pi * k * x) ** 2
    d2 = lambda x, k: math.pi * k * np.sin(2.0 * math.pi * k * x)
    for a, b in [(0, 1)] if nd == 2 else [(0, 1), (0, 2), (1, 2)]:
        for _ in range(2):
            k, l, w = rng.integers(1, 4), rng.integers(1, 4), amplitude * rng.uniform(-0.2, 0.2)
            rest = np.ones(X.shape[0])
            for c in range(nd):
                if c not in (a, b):
                    rest = rest * s2(X[:, c], 1)
            f[:, a] += w * s2(X[:, a], k) * d2(X[:, b], l) * rest / (math.pi * l)
            f[:, b] -= w * d2(X[:, a], k) * s2(X[:, b], l) * rest / (math.pi * k)
    for c in range(nd):
        f[:, nd] += amplitude * rng.uniform(-0.05, 0.05) * (np.cos(math.pi * X[:, c]) - 1.0)
    return f


def _states(case, mesh, seed):
    """u_{n-1}, u_n, their rate, and the ramp factor of the step to come.  Cavities are inside the lid's ramp, so
    the step moves the boundary too; the wake carries its full inflow."""
    rng = np.random.default_rng(seed)
    X = mesh.coords
    if case["mesh"] == "wake":
        r = np.hypot(X[:, 0], X[:, 1])
        th = np.arctan2(X[:, 1], X[:, 0])
        near = 1.0 - np.exp(-(r - 0.5) / 0.2)
        u = np.zeros((len(r), 3))
        u[:, 0] = near * (1.0 - 0.25 * np.cos(2.0 * th) / r ** 2)
        u[:, 1] = -near * 0.25 * np.sin(2.0 * th) / r ** 2
        u[:, 2] = 0.5 * (1.0 - u[:, 0] ** 2 - u[:, 1] ** 2) * np.exp(-(r - 0.5))
        w = near * np.exp(-0.1 * r)
        rate = np.zeros_like(u)
        for _ in range(3):
            k, a, b = rng.integers(1, 4), rng.uniform(-0.1, 0.1), rng.uniform(0, 2 * math.pi)
            u[:, 1] += a * w * np.cos(k * th + b)
            rate[:, 1] += 0.2 * a * w * np.sin(k * th + b)
        level, ramp = 1.0, 1.0
    else:
        u, rate = _modes(X, rng, 1.0), _modes(X, rng, 0.2)
        level, ramp = 0.5, 0.6
    d = mesh.dbc
    free = np.ones((mesh.nNode, mesh.ndof), dtype=bool)
    g = (d[:, 0].astype(np.int64), d[:, 1].astype(np.int64))
    free[g] = False
    u[g] = level * d[:, 2]
    rate[g] = (ramp - level) / 0.1 * d[:, 2]
    before = u - 0.1 * rate * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, u.shape) * free)
    return before.ravel(), u.ravel(), rate.ravel(), ramp


def _control(case, re=None):
    return meshgen.control_for(1000, 0.05 if case["work"] == "batch" else 0.1, 1.0 / float(case["re"] if re is None else re))


def _solver(case):
    if case.get("precision") == "mixed":
        return dict(precision="mixed", ksp="gmres", restart=case["restart"], pc=case["pc"], ilu_levels=case["levels"],
                    inner_restart=20, inner_rtol=1e-2, refine_rtol=1e-14, refine_atol=-1.0, max_it=2000)
    ksp = case.get("ksp", "gmres")
    return dict(ksp=ksp, pc=case["pc"], ilu_levels=case.get("levels", 0), restart=case["restart"],
                rtol=1e-15 if ksp == "bcgs" else 1e-14, max_it=40000)


def _batch_cases(case):
    """The cavities of a batch: sides spread evenly over n..n_hi, Reynolds numbers over 100..1000."""
    k = max(case["count"] - 1, 1)
    out = []
    for i in range(case["count"]):
        n = case["n"] + (case["n_hi"] - case["n"]) * i // k
        mesh = meshgen.cavity2d(n)
        out.append((mesh, _control(case, re=100.0 * 10.0 ** (((7 * i) % (k + 1)) / (k + 1)))))
    return out


def _net_params(seed):
    """Weights of the size that training starts from: uniform, +-gain sqrt(3 / inputs); biases small."""
    rng = np.random.default_rng([seed, 77])
    p = []
    for k, no, gain in [(FIN, HID, 1.0)] + [(2 * HID, HID, 0.5)] * LAYERS + [(HID, FOUT, 0.5)]:
        p += [gain * math.sqrt(3.0 / k) * rng.uniform(-1.0, 1.0, k * no), 0.05 * rng.uniform(-1.0, 1.0, no)]
    return np.concatenate(p).astype(np.float32)


def _net_scales(ndof):
    return np.concatenate([np.full(ndof, 0.2), np.full(ndof, 0.05)]).astype(np.float32), np.full(ndof, 0.01, np.float32)


def _net_sample(case, mesh, seed):
    """u_{n-1}, u_n, u_{n+1}: two smooth increments, prescribed dofs at rest."""
    before, u, rate, _ = _states(case, mesh, seed)
    rng = np.random.default_rng([seed, 5])
    bend = _modes(mesh.coords, rng, 0.05)
    d = mesh.dbc
    bend[d[:, 0].astype(np.int64), d[:, 1].astype(np.int64)] = 0.0
    return before, u, u + (u - before) + bend.ravel()


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64))
    return t.pin_memory() if torch.cuda.is_available() else t


def prepare(case, seed):
    if case["work"] == "net":
        mesh = _mesh(case)
        h = Handle(mesh, meshgen.control_for(10, 0.1, 0.01), restart=2)
        net = Mpnn(h, seed=0)
        net.set_scales(*_net_scales(mesh.ndof))
        net.set_params(_net_params(seed))
        net.add_sample(*_net_sample(case, mesh, seed))
        return {"case": case, "net": net, "handle": h}
    if case["work"] == "batch":
        pairs = _batch_cases(case)
        b = Batch(pairs, **_solver(case))
        b.set_schedule(len(pairs), 4, 1)
        st = [_states(case, m, [seed, i]) for i, (m, _) in enumerate(pairs)]
        return {"case": case, "batch": b, "ramp": st[0][3], "u": [_pinned(s[1]) for s in st],
                "rate": [s[2] for s in st], "out": [_pinned(np.zeros_like(s[1])) for s in st]}
    mesh = _mesh(case)
    h = Handle(mesh, _control(case), **_solver(case))
    before, u, rate, ramp = _states(case, mesh, seed)
    state = {"case": case, "handle": h, "u": _pinned(u), "before": _pinned(before), "rate": _pinned(rate), "ramp": ramp,
             "out": _pinned(np.zeros_like(u))}
    if case["guess"] == "extrapolation":
        h.set_guess_mode(("extrapolation",))
    elif case["guess"] == "network":
        net = Mpnn(h, seed=0)
        net.set_scales(*_net_scales(mesh.ndof))
        net.set_params(_net_params(seed))
        net.attach(("network", "extrapolation"))
        state["net"] = net
    return state


def run(state):
    """One pass.  A step starts from the state's u_n with its history, so passes repeat the same step."""
    work = state["case"]["work"]
    if work == "net":
        loss, grad = state["net"].loss_grad(0)
        return {"loss": np.float32(loss), "gradient": grad}
    if work == "batch":
        b = state["batch"]
        for h, u, rate in zip(b.handles, state["u"], state["rate"]):
            h.set_solution_ptr(u.data_ptr())
            h.set_history(None, rate)
        b.step([state["ramp"]] * len(b))
        for h, o in zip(b.handles, state["out"]):
            h.get_solution_ptr(o.data_ptr())
        return state["out"]
    h = state["handle"]
    h.set_solution_ptr(state["u"].data_ptr())
    h.set_history(state["before"].numpy(), state["rate"].numpy())
    h.step(state["ramp"], state["ramp"])
    h.get_solution_ptr(state["out"].data_ptr())
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _pattern_blocks(mesh):
    """Node pairs that share an element."""
    a = mesh.conn.astype(np.int64)
    return int(torch.unique(torch.from_numpy((a[:, :, None] * mesh.nNode + a[:, None, :]).ravel())).numel())


def work(case):
    """A step has to read the mesh and three state vectors, write the matrix (assembly), read it once for the
    solve and write the solution; the operations are those of one assembly and one product.  (How often a Krylov
    method reads the matrix again is the method's affair.)  The network reads its inputs, the node graph and its
    weights and writes the gradient; its operations are those of the dense layers, forward and twice backward."""
    if case["work"] == "net":
        mesh = _mesh(case)
        blocks, N = _pattern_blocks(mesh), mesh.nNode
        dense = FIN * HID + LAYERS * 2 * HID * HID + HID * FOUT
        return {"bytes": N * (2 * FIN + 8 * FOUT) + 4.0 * blocks + 8.0 * NET_PARAMS, "flops": 6.0 * N * dense}
    meshes = [m for m, _ in _batch_cases(case)] if case["work"] == "batch" else [_mesh(case)]
    nbytes = flops = 0.0
    for m in meshes:
        bb, V = m.ndof ** 2, 8.0 * m.nNode * m.ndof
        B = _pattern_blocks(m)
        nbytes += 2.0 * 8.0 * B * bb + 8.0 * m.coords.size + 4.0 * m.conn.size + 4.0 * B + 4.0 * V
        points = {8: 8, 4: 4 if m.ndim == 2 else 1, 3: 1}[m.npElem]
        flops += 2.0 * B * bb + 6.0 * bb * m.nElem * m.npElem ** 2 * points
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch alone

def _basis(npe, ndim):
    """Quadrature weights, basis values and reference derivatives: (G,), (G, npe), (G, ndim, npe)."""
    q = 0.577350269189626
    if npe == 8:
        pts = [[q if g & 1 << c else -q for c in range(3)] for g in range(8)]
        w, N, D = [], [], []
        for x, y, z in pts:
            a, b, c = (1 - x, 1 + x), (1 - y, 1 + y), (1 - z, 1 + z)
            o = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
            w.append(1.0)
            N.append([0.125 * a[i] * b[j] * c[k] for i, j, k in o])
            # the second derivative row pairs nodes (2, 3) and (6, 7) with the factors in this order, as the solver does
            D.append([[(-1, 1)[i] * 0.125 * b[j] * c[k] for i, j, k in o],
                      [(-1, 1)[j] * 0.125 * a[m] * c[k] for (i, j, k), m in zip(o, (0, 1, 0, 1) * 2)],
                      [(-1, 1)[k] * 0.125 * a[m] * b[j] for (i, j, k), m in zip(o, (0, 1, 0, 1) * 2)]])
        return w, N, D
    if npe == 4 and ndim == 2:
        w, N, D = [], [], []
        for g in range(4):
            x, y = q if g & 1 else -q, q if g & 2 else -q
            a, b = (0.5 * (1 - x), 0.5 * (1 + x)), (0.5 * (1 - y), 0.5 * (1 + y))
            w.append(1.0)
            N.append([b[0] * a[0], b[0] * a[1], b[1] * a[1], b[1] * a[0]])
            D.append([[-0.5 * b[0], 0.5 * b[0], 0.5 * b[1], -0.5 * b[1]], [-0.5 * a[0], -0.5 * a[1], 0.5 * a[1], 0.5 * a[0]]])
        return w, N, D
    if npe == 4:
        return [1.0 / 6.0], [[0.25] * 4], [[[-1, 1, 0, 0], [-1, 0, 1, 0], [-1, 0, 0, 1]]]
    return [4.0], [[1.0, 0.0, 0.0]], [[[-1, 1, 0], [-1, 0, 1]]]


def _exact_step(mesh, ctrl, u, rate, ramp):
    """One semi-implicit generalised-alpha step.  The residual is affine in the new state, so the step is one
    linear solve: stabilised element matrices, dense assembly, LU."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)
    nd, npe, ndof = mesh.ndim, mesh.npElem, mesh.ndof
    rho, mu, dt = ctrl.rho, ctrl.mu, ctrl.dt
    ri = ctrl.rhoInf
    af, am = 1.0 / (1.0 + ri), 0.5 * (3.0 - ri) / (1.0 + ri)
    gam = 0.5 + am - af
    acc = am / gam / dt
    flip = -1.0 if npe == 8 else 1.0
    ci = 10.0 if nd == 3 else 4.0
    conn = torch.as_tensor(mesh.conn.astype(np.int64), device=dev)
    w, N, D = (T(a) for a in _basis(npe, nd))
    X = T(mesh.coords)[conn]
    prev = T(u).reshape(-1, ndof)[conn]
    dot0 = T(rate).reshape(-1, ndof)
    new_dot = (1.0 - 1.0 / gam) * dot0                      # at the constant predictor u_{n+1} = u_n
    vdot = (am * new_dot + (1.0 - am) * dot0)[conn]
    B = torch.einsum("gam,emc->egac", D, X)                 # rows: reference derivative a of coordinate c
    J = torch.linalg.det(B)
    dN = torch.einsum("egca,gai->egci", torch.linalg.inv(B), D)
    dvol = w * J
    vol = dvol.sum(1).abs()
    h = torch.sqrt(4.0 * vol / math.pi) if nd == 2 else (6.0 * vol / math.pi) ** (1.0 / 3.0)
    G = (4.0 / h / h)[:, None]
    vel, pres = prev[..., :nd], prev[..., nd]
    v = torch.einsum("gi,eia->ega", N, vel)
    g = torch.einsum("egci,eia->egac", dN, vel)
    p, dp = pres @ N.T, torch.einsum("egci,ei->egc", dN, pres)
    a = torch.einsum("gi,eia->ega", N, vdot[..., :nd])
    conv = torch.einsum("egac,egc->ega", g, v)
    tau = 1.0 / torch.sqrt((v * v).sum(-1) * G + ci * (mu / rho) ** 2 * nd * G * G) / rho
    t_su, t_ps = tau * ctrl.stab[0], tau * ctrl.stab[1]
    res = rho * (a + conv)
    strong = res + dp
    eye = torch.eye(nd, dtype=torch.float64, device=dev)
    sig = mu * g - p[..., None, None] * eye
    Nd = N[None] * dvol[..., None]
    Bd = dN * dvol[..., None, None]
    F = torch.zeros(*conn.shape, ndof, dtype=torch.float64, device=dev)
    F[..., :nd] = -torch.einsum("egi,ega->eia", Nd, res) - torch.einsum("egci,egac->eia", Bd, sig)
    F[..., nd] = -flip * (torch.einsum("egi,eg->ei", Nd, g.diagonal(dim1=-2, dim2=-1).sum(-1))
                          + torch.einsum("egai,eg,ega->ei", Bd, t_ps, strong))
    Da = rho * torch.einsum("ega,egai->egi", v, Bd) * t_su[..., None] if nd == 2 else None
    Db = rho * torch.einsum("ega,egaj->egj", v, dN)
    K = torch.zeros(mesh.nElem, npe, ndof, npe, ndof, dtype=torch.float64, device=dev)
    # per point: advection matrix A[a, c, j] = rho (N_j du_a/dx_c + delta v . grad N_j)
    A = rho * torch.einsum("egac,gj->egacj", g, N) + torch.einsum("egj,ac->egacj", Db, eye)
    M = rho * acc * torch.einsum("gj,ac->gacj", N, eye)
    dif = mu * af * torch.einsum("egbi,egbj->eij", Bd, dN)
    K[:, :, :nd, :, :nd] = (af * torch.einsum("egi,egacj->eiajc", Nd, A) + torch.einsum("egi,gacj->eiajc", Nd, M)
                            + torch.einsum("eij,ac->eiajc", dif, eye))
    K[:, :, :nd, :, nd] = -af * torch.einsum("egai,gj->eiaj", Bd, N)
    op = af * A + M[None]                                   # momentum operator of the stabilisation terms
    K[:, :, nd, :, :nd] = flip * (af * torch.einsum("egi,egcj->eijc", Nd, dN)
                                  + torch.einsum("eg,egai,egacj->eijc", t_ps, Bd, op))
    K[:, :, nd, :, nd] = flip * af * torch.einsum("eg,egai,egaj->eij", t_ps, Bd, dN)
    if Da is not None:
        F[..., :nd] -= torch.einsum("egi,ega->eia", Da, strong)
        K[:, :, :nd, :, :nd] += torch.einsum("egi,egacj->eiajc", Da, op)
        K[:, :, :nd, :, nd] += af * torch.einsum("egi,egaj->eiaj", Da, dN)
    n = mesh.nNode * ndof
    dof = (conn[..., None] * ndof + torch.arange(ndof, device=dev)).reshape(mesh.nElem, -1)
    k = dof.shape[1]
    full = torch.zeros(n * n, dtype=torch.float64, device=dev)
    full.index_put_(((dof[:, :, None] * n + dof[:, None, :]).reshape(-1),), K.reshape(-1), accumulate=True)
    full = full.reshape(n, n)
    rhs = torch.zeros(n, dtype=torch.float64, device=dev)
    rhs.index_put_((dof.reshape(-1),), F.reshape(mesh.nElem, k).reshape(-1), accumulate=True)
    fixed = torch.as_tensor((mesh.dbc[:, 0] * ndof + mesh.dbc[:, 1]).astype(np.int64), device=dev)
    step = torch.zeros(n, dtype=torch.float64, device=dev)
    step[fixed] = T(mesh.dbc[:, 2]) * ramp - T(u)[fixed]
    free = torch.ones(n, dtype=torch.bool, device=dev)
    free[fixed] = False
    rhs = (rhs - full @ step)[free]
    full = full[free][:, free]
    d = torch.linalg.solve(full, rhs)
    d = d + torch.linalg.solve(full, rhs - full @ d)
    step[free] = d
    return (T(u) + step).cpu()


def _exact_net(case, seed):
    """Loss and gradient of the network in 64 bits, no rounding of weights or activations."""
    mesh = _mesh(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)
    nd, ndof, n = mesh.ndim, mesh.ndof, mesh.nNode
    um, u, up = (T(a).reshape(n, ndof) for a in _net_sample(case, mesh, seed))
    s_in, s_out = (T(a) for a in _net_scales(ndof))
    X = T(mesh.coords)
    lo, hi = X.min(0).values, X.max(0).values
    f = torch.zeros(n, FIN, dtype=torch.float64, device=dev)
    f[:, :ndof] = u / s_in[:ndof]
    f[:, ndof:2 * ndof] = (u - um) / s_in[ndof:]
    f[:, 2 * ndof:2 * ndof + nd] = 2.0 * (X - lo) / (hi - lo) - 1.0
    target = ((up - u) - (u - um)) / s_out
    mask = torch.ones(n, ndof, dtype=torch.float64, device=dev)
    mask[torch.as_tensor(mesh.dbc[:, 0].astype(np.int64), device=dev),
         torch.as_tensor(mesh.dbc[:, 1].astype(np.int64), device=dev)] = 0.0
    a = torch.as_tensor(mesh.conn.astype(np.int64), device=dev)
    pairs = torch.unique((a[:, :, None] * n + a[:, None, :]).reshape(-1))
    row, col = pairs // n, pairs % n
    deg = torch.bincount(row, minlength=n).double()[:, None]
    params = T(_net_params(seed)).requires_grad_(True)
    o = 0

    def take(*shape):
        nonlocal o
        k = math.prod(shape)
        o += k
        return params[o - k:o].reshape(shape)

    h = torch.relu(f @ take(FIN, HID) + take(HID))
    for _ in range(LAYERS):
        mean = torch.zeros_like(h).index_add_(0, row, h[col]) / deg
        h = h + torch.relu(torch.cat([h, mean], 1) @ take(2 * HID, HID) + take(HID))
    y = (h @ take(HID, FOUT) + take(FOUT))[:, :ndof]
    loss = (((y - target) * mask) ** 2).sum() / mask.sum()
    loss.backward()
    return {"loss": loss.detach().cpu(), "gradient": params.grad.cpu()}


def exact(case, seed):
    if case["work"] == "net":
        return _exact_net(case, seed)
    if case["work"] == "batch":
        pairs = _batch_cases(case)
        if max(m.nNode * m.ndof for m, _ in pairs) > DENSE_LIMIT:
            return None
        out = []
        for i, (m, c) in enumerate(pairs):
            _, u, rate, ramp = _states(case, m, [seed, i])
            out.append(_exact_step(m, c, u, rate, ramp))
        return out
    mesh = _mesh(case)
    if mesh.nNode * mesh.ndof > DENSE_LIMIT:
        return None          # too large for a dense factorisation in a few seconds
    _, u, rate, ramp = _states(case, mesh, seed)
    return _exact_step(mesh, _control(case), u, rate, ramp)
