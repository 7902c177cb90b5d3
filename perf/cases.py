"""The work that programs built on cfd_gb300 have it do, as cases for a timing harness.

A case is a dict of plain values.  `kind` says which public entry points it runs through:

    march    the resident context's time loop, one print interval: `steps` steps, then the
             state into the program's page-locked buffers (cfd_step, cfd_ctx_download_state)
    coupled  a host program that owns U: upload of U, one step, download of U, every step
    bicg     the drop-in biCG on host arrays, a cold mesh-motion solve
    calcrhs  the drop-in calcRHS on host arrays
    infer    the learned guess of a mesh motion (Net.forward, BF16)
    train    loss and gradient of the learned guess on one mesh (Net.loss_grad, FP32)

The meshes are the package's seeded O-grids (nr rings of ntheta nodes); the flow and the
motion are those of its workloads (cylinder at Mach 0.3, ellipse at Mach 0.8).
"""
import ctypes
import math

import numpy as np
import torch

from cfd_gb300 import abi, case as cs, learned, solver

# ranges of the drawn cases: nodes of the mesh, by kind (and precision of a march)
RANGES = {"march fp64": (2.0e3, 3.0e5), "march mixed": (4.0e3, 1.2e6), "coupled": (5.0e4, 1.0e6),
          "bicg": (8.0e3, 2.7e5), "calcrhs": (8.0e3, 5.0e5), "infer": (3.0e4, 1.1e6),
          "train": (8.0e3, 7.0e4)}


def listed():
    return [
        # the reference's own CPU-sized run: small mesh that does not move, plain FP64
        dict(name="fp64_cylinder_8k", kind="march", precision="fp64", body="cylinder", nr=64,
             ntheta=128, motion="none", guess="previous", test="abs", steps=10),
        # the plain form with the moving mesh, odd ring count, heaving cylinder
        dict(name="fp64_heave_69k", kind="march", precision="fp64", body="cylinder", nr=257,
             ntheta=270, motion="heave", guess="extrapolated", test="abs", steps=5),
        # the plain form at the size the throughput is quoted on
        dict(name="fp64_ellipse_1M", kind="march", precision="fp64", body="ellipse", nr=1024,
             ntheta=1024, motion="heave", guess="previous", test="abs", steps=2),
        # the mixed form on a small mesh: launches and latency
        dict(name="mixed_ellipse_15k", kind="march", precision="mixed", body="ellipse", nr=101,
             ntheta=150, motion="heave", guess="previous", test="abs", steps=20),
        # the mixed form under the relative BiCG test with the refined learned guess
        dict(name="mixed_relative_262k", kind="march", precision="mixed", body="ellipse", nr=512,
             ntheta=512, motion="heave", guess="refined", test="rel", steps=20),
        # the headline run: mixed form with the learned guess, one million nodes
        dict(name="mixed_learned_1M", kind="march", precision="mixed", body="ellipse", nr=1024,
             ntheta=1024, motion="heave", guess="learned", test="abs", steps=20),
        # the largest mesh, heave and pitch, twice as many rings as nodes in a ring
        dict(name="mixed_pitch_3M", kind="march", precision="mixed", body="ellipse", nr=2049,
             ntheta=1536, motion="pitch", guess="extrapolated", test="abs", steps=10),
        # a host code that keeps U itself and calls the step
        dict(name="coupled_mixed_590k", kind="coupled", precision="mixed", body="ellipse", nr=768,
             ntheta=768, motion="heave", guess="learned", test="abs", steps=4),
        # the first mesh-motion solve of a run, or one solve of a training set
        dict(name="bicg_cold_147k", kind="bicg", body="ellipse", nr=384, ntheta=384),
        # one reference routine replaced in a host code
        dict(name="calcrhs_host_262k", kind="calcrhs", body="cylinder", nr=512, ntheta=512),
        # the learned guess on the headline mesh
        dict(name="infer_bf16_1M", kind="infer", body="ellipse", nr=1024, ntheta=1024),
        # one mesh of the training set
        dict(name="train_grad_50k", kind="train", body="ellipse", nr=193, ntheta=258),
    ]


def _grid(rng, lo, hi):
    """(nr, ntheta) of a mesh with log-uniformly drawn node count; ntheta is even."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = math.exp(rng.uniform(math.log(0.6), math.log(1.7)))
    ntheta = max(16, 2 * round(math.sqrt(n * aspect) / 2))
    return max(12, round(n / ntheta)), ntheta


def draw(rng):
    kind = rng.choice(["march fp64", "march mixed", "march mixed", "coupled", "bicg", "calcrhs",
                       "infer", "train"])
    nr, ntheta = _grid(rng, *RANGES[kind])
    c = dict(kind=kind.split()[0], body=rng.choice(["cylinder", "ellipse"]), nr=nr, ntheta=ntheta)
    if kind == "march fp64":
        c.update(precision="fp64", body="cylinder", motion=rng.choice(["none", "heave"]),
                 guess=rng.choice(["previous", "extrapolated"]), test="abs",
                 steps=rng.randint(1, 5))
    elif kind == "march mixed":
        test = rng.choice(["abs", "abs", "rel"])
        c.update(precision="mixed", body="ellipse", test=test,
                 motion="heave" if test == "rel" else rng.choice(["heave", "pitch"]),
                 guess="refined" if test == "rel" else rng.choice(["extrapolated", "learned"]),
                 steps=rng.randint(2, 20))
    elif kind == "coupled":
        c.update(precision="mixed", body="ellipse", motion="heave", test="abs",
                 guess=rng.choice(["previous", "learned"]), steps=rng.randint(1, 4))
    return c


# ------------------------------------------------------------------ meshes and programs
def _mesh(c, seed):
    mixed = c.get("precision") == "mixed"
    kw = dict(moving=0 if c.get("motion") == "none" else 1, motion_law=abi.CFD_MOTION_HARMONIC)
    if c["body"] == "cylinder":
        if kw["moving"]:
            kw.update(heave_amp=0.2, motion_freq=0.2, mass_mode=abi.CFD_MASS_GCL_CORRECTED)
        p = cs.flow_params(0.3, 200.0 if kw["moving"] else 100.0, **kw)
        k = cs.ogrid_case("cylinder", c["nr"], c["ntheta"], p, "cylinder", r_out=20.0, seed=seed)
    else:
        kw.update(heave_amp=0.05, motion_freq=0.1, mass_mode=abi.CFD_MASS_GCL_CORRECTED)
        if c.get("motion") == "pitch":
            kw["pitch_amp"] = math.radians(3.0)
        p = cs.flow_params(0.8, 5000.0, fsafe=0.25, **kw)
        k = cs.ogrid_case("ellipse", c["nr"], c["ntheta"], p, "ellipse", incidence_deg=2.0,
                          r_out=30.0, seed=seed)
    p.estab_mode = abi.CFD_ESTAB_REGULARIZED if mixed else abi.CFD_ESTAB_REFERENCE
    if c.get("test") == "rel":
        p.bicg_tol_mode, p.bicg_maxit = abi.CFD_BICG_TOL_REL, 20000
    p.guess_mode = {"previous": abi.CFD_GUESS_PREVIOUS, "extrapolated": abi.CFD_GUESS_EXTRAPOLATED,
                    "learned": abi.CFD_GUESS_LEARNED,
                    "refined": abi.CFD_GUESS_LEARNED_EXTRAPOLATED}[c.get("guess", "previous")]
    return k


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _march(c, seed):
    k = _mesh(c, seed)
    s = solver.Solver(k, abi.CFD_PREC_MIXED if c["precision"] == "mixed" else abi.CFD_PREC_FP64)
    st = dict(c=c, solver=s, U=_pinned(k.npoin, 4), T=_pinned(k.npoin), X=_pinned(k.npoin),
              Y=_pinned(k.npoin))
    if c["guess"] in ("learned", "refined"):
        st["net"] = learned.Net.load()
        s.set_guess_net(st["net"])
        s.set_guess_refine(c["guess"] == "refined")
    s.step(3)  # the run is under way: its cold mesh-motion solve and start-up are behind it
    if c["kind"] == "coupled":
        _download(st, "U")
    return st


def _download(st, what):
    p = [_ptr(st[q]) if q in what else None for q in "UTXY"]
    abi.check(abi.lib().cfd_ctx_download_state(st["solver"].h, *p), "cfd_ctx_download_state")
    return {q: st[q] for q in what}


def _rigid(k, rng):
    return learned.rigid_bc(k, float(rng.uniform(0.05, 0.3)), float(rng.uniform(2.0, 10.0)))


def _bicg(c, seed):
    k = _mesh(c, seed)
    lap = learned.Laplace(k)
    gx, gy = _rigid(k, np.random.default_rng(seed))
    return dict(c=c, vals=lap.vals, idx=lap.idx, rp=lap.rp, diag=lap.diag, fix=gy,
                node=lap.bnode, x0=np.zeros(k.npoin), b=np.zeros(k.npoin))


def _rhs_inputs(c, seed):
    """Host arrays of a calcRHS call: a smoothly and randomly perturbed freestream."""
    k = _mesh(c, seed)
    p, rng = k.params, np.random.default_rng(seed)
    f = 0.05 * np.sin(k.x + 0.3 * k.y + rng.uniform(0, 6)) + 0.01 * rng.uniform(-1, 1, k.npoin)
    rho, T = p.rho_inf * (1 + f), p.t_inf * (1 - 0.5 * f)
    u, v = p.u_inf * (1 + 0.3 * f), 0.2 * p.u_inf * f
    U = np.stack([rho, rho * u, rho * v, rho * (p.fcv * T + 0.5 * (u * u + v * v))], 1)
    g = solver.deriv(k.x, k.y, k.inpoel)
    W = np.zeros(k.npoin)
    dt, _ = solver.deltat(T, u, v, W, W, g["area"], k.inpoel, p.fsafe, p.fr, p.gama, p.t_inf)
    est = solver.ESTAB(U, T, np.full(k.npoin, p.gama), u, v, W, W, g["dNx"], g["dNy"], k.inpoel,
                       p.gama, p.fr, float(dt.min()), p.rho_inf, p.t_inf)
    return dict(c=c, U=U, T=T, dNx=g["dNx"], dNy=g["dNy"], area=g["area"], est=est, dtl=dt,
                inpoel=k.inpoel, gas=p.gas6(), rhs=np.zeros((k.npoin, 4)))


def _graph(c, seed):
    k = _mesh(c, seed)
    st = dict(c=c, net=learned.Net.load(), graph=learned.Graph(k))
    if c["kind"] == "infer":
        st["graph"].set_bc(*_rigid(k, np.random.default_rng(seed)))
    else:
        st["graph"].set_target(*_targets(k, seed))
    return st


def _targets(k, seed):
    """Smooth fields that fall from the body to the outer boundary, as the solves' do."""
    rng = np.random.default_rng(seed)
    r, th = np.hypot(k.x, k.y), np.arctan2(k.y, k.x)
    phi = np.clip(1.0 - np.log(np.maximum(r, 0.5) / 0.5) / np.log(r.max() / 0.5), 0.0, 1.0)
    a, b = rng.uniform(0.3, 0.6, 2)
    return phi, a * phi ** 2 * np.cos(th), b * phi ** 2 * np.sin(th)


def prepare(case, seed):
    return {"march": _march, "coupled": _march, "bicg": _bicg, "calcrhs": _rhs_inputs,
            "infer": _graph, "train": _graph}[case["kind"]](case, int(seed))


def run(state):
    c = state["c"]
    if c["kind"] == "march":
        state["solver"].step(c["steps"])
        return _download(state, "UTXY")
    if c["kind"] == "coupled":
        s = state["solver"]
        for _ in range(c["steps"]):
            abi.check(abi.lib().cfd_ctx_upload_state(s.h, _ptr(state["U"]), None, None, None),
                      "cfd_ctx_upload_state")
            s.step(1)
            _download(state, "U")
        return {"U": state["U"]}
    if c["kind"] == "bicg":
        x, info = solver.biCG(state["vals"], state["idx"], state["rp"], state["diag"],
                              state["x0"], state["b"], state["fix"], state["node"], maxit=20000)
        return {"x": x, "iters": int(info.iters)}
    if c["kind"] == "calcrhs":
        s = state
        s["rhs"][:] = 0.0  # the caller zeroes what calcRHS adds to
        return solver.calcRHS(s["rhs"], s["U"], None, s["dNx"], s["dNy"], s["area"], s["est"][0],
                              s["dtl"], *s["est"][1:], s["inpoel"], s["T"], s["gas"])
    if c["kind"] == "infer":
        return state["net"].forward(state["graph"], bf16=True)
    loss, grad = state["net"].loss_grad(state["graph"])
    return {"loss": loss, "grad": grad}


def work(case):
    n, kind = float(case["nr"] * case["ntheta"]), case["kind"]
    e = 2.0 * n  # triangles; 7 matrix entries a row, 6 neighbours a node
    if kind in ("march", "coupled"):
        # per step: U, T, velocities, X, Y, W, M and the increments read and written once,
        # the connectivity read once; deltat, ESTAB, calcRHS with its stages, the geometry
        steps = case["steps"]
        out = 64.0 * n * (steps if kind == "coupled" else 1)
        return {"bytes": steps * (2 * 14 * 8 * n + 12 * e) + out, "flops": steps * 2300.0 * e}
    if kind == "bicg":  # about 3.4 sqrt(n) iterations of a product and five vector updates
        it = 3.4 * math.sqrt(n)
        return {"bytes": n * (7 * 12 + 4 + 8 * 5), "flops": it * n * (14 + 14)}
    if kind == "calcrhs":
        return {"bytes": 8 * (4 * n * 3 + n) + e * (8 * 12 + 12), "flops": 1100.0 * e}
    dense = 2 * (64 * 10 + 4 * (64 * 128 + 128 * 64) + 3 * 64)
    edge = 4 * 6 * 64 * 9
    if kind == "infer":
        return {"bytes": n * (16 + 28 + 16), "flops": n * (dense + edge)}
    return {"bytes": n * (16 + 28 + 24) + 2 * 4 * 67715, "flops": 3 * n * (dense + edge)}


# ------------------------------------------------------------------ the same in 64 bits
def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda" if torch.cuda.is_available()
                           else "cpu")


def _exact_bicg(s):
    """The solve to (nearly) the last bit: Jacobi-PCG on the free rows, restarted from the
    true residual.  The iteration count has no value of its own."""
    n = len(s["x0"])
    A = torch.sparse_csr_tensor(_t(s["rp"]), _t(s["idx"] - 1), _t(s["vals"]), (n, n))
    x = _t(s["x0"]).clone()
    fix = _t(s["node"].astype(np.int64) - 1)
    x[fix] = _t(s["fix"])
    free = torch.ones_like(x)
    free[fix] = 0.0
    d, b = _t(s["diag"]), _t(s["b"])
    for _ in range(3):
        r = (b - A @ x) * free
        z = r / d
        p, rz = z.clone(), r @ z
        stop = float(r @ r) * 1e-24
        for it in range(int(8 * math.sqrt(n)) + 200):
            q = (A @ p) * free
            a = rz / (p @ q)
            x += a * p
            r -= a * q
            z = r / d
            rz, old = r @ z, rz
            if it % 50 == 0 and not float(r @ r) > stop:
                break
            p = z + (rz / old) * p
    return {"x": x.cpu().numpy(), "iters": None}


def _exact_rhs(s):
    """calcRHS of linear triangles with three edge-midpoint quadrature points."""
    cv, lam_ref, mu_ref, g, t_inf, cte = (float(v) for v in s["gas"])
    el = _t(s["inpoel"].astype(np.int64) - 1)
    N = [_t(s["dNx"]), _t(s["dNy"])]
    Un = _t(s["U"])[el]
    G = [torch.einsum("eiq,ei->eq", Un, d) for d in N]  # Ux, Uy
    ta = _t(s["T"])[el].mean(1)
    visc = [ref * (ta / t_inf) ** 1.5 * (t_inf + k) / (ta + k)
            for ref, k in ((mu_ref, 110.0), (lam_ref, 194.0))]
    tau = torch.stack([_t(t) for t in s["est"][1:]], 1)
    nu = _t(s["est"][0]) * cte
    r = torch.zeros_like(Un)
    for k in range(3):
        Uk = 0.5 * (Un.sum(1) - Un[:, k])
        rho = Uk[:, 0]
        v = [Uk[:, 1] / rho, Uk[:, 2] / rho]
        ev, V = Uk[:, 3] / rho, v[0] ** 2 + v[1] ** 2

        def jac(d, X):  # the inviscid flux Jacobian of direction d times X
            m, o = 1 + d, 2 - d
            w = [None] * 4
            w[0] = X[:, m]
            w[m] = ((0.5 * (g - 1) * V - v[d] ** 2) * X[:, 0] + (3 - g) * v[d] * X[:, m]
                    - (g - 1) * v[1 - d] * X[:, o] + (g - 1) * X[:, 3])
            w[o] = -v[0] * v[1] * X[:, 0] + v[1 - d] * X[:, m] + v[d] * X[:, o]
            w[3] = (v[d] * ((g - 1) * V - g * ev) * X[:, 0]
                    + (g * ev - 0.5 * (g - 1) * V - (g - 1) * v[d] ** 2) * X[:, m]
                    - (g - 1) * v[0] * v[1] * X[:, o] + g * v[d] * X[:, 3])
            return torch.stack(w, 1)

        A = jac(0, G[0]) + jac(1, G[1])
        B = [jac(0, A), jac(1, A)]
        # velocity and temperature-like gradients of the viscous flux
        dv = [[(G[b][:, 1 + a] - v[a] * G[b][:, 0]) / rho for b in (0, 1)] for a in (0, 1)]
        de = [(G[b][:, 3] - ev * G[b][:, 0]) / rho - v[0] * dv[0][b] - v[1] * dv[1][b]
              for b in (0, 1)]
        mu, lam = visc
        div = (dv[0][0] + dv[1][1]) * (2.0 / 3.0)
        K = []
        for b in (0, 1):
            t = [mu * (dv[a][b] + dv[b][a] - (div if a == b else 0.0)) for a in (0, 1)]
            K.append(torch.stack([torch.zeros_like(mu), t[0], t[1],
                                  v[0] * t[0] + v[1] * t[1] + lam / cv * de[b]], 1))
        for i in range(3):
            if i != k:
                r[:, i] += 0.5 * A
            r[:, i] += sum(N[d][:, i:i + 1] * (tau[:, i:i + 1] * B[d] + nu[:, None] * G[d] + K[d])
                           for d in (0, 1))
    r *= (_t(s["area"]) * _t(s["dtl"]) / 3.0)[:, None, None]
    out = torch.zeros_like(_t(s["U"]))
    out.index_add_(0, el.reshape(-1), r.reshape(-1, 4))
    return out.cpu().numpy()


def _net64(k, gx, gy):
    """(forward function of the flat FP64 weights -> y, globals) on the case's mesh."""
    x, y = _t(k.x), _t(k.y)
    body, outer = _t(k.i_m.astype(np.int64) - 1), _t(k.ifm.astype(np.int64) - 1)
    cx, cy = x[body].mean(), y[body].mean()
    dx, dy = x - cx, y - cy
    r = torch.hypot(dx, dy)
    L, R = 2 * r[body].max(), r[outer].mean()
    D = torch.stack([dx[body], dy[body]], 1)
    S = D.T @ D
    nb = len(k.i_m)
    hx, mxy, tr = (S[0, 0] - S[1, 1]) / (2 * nb), S[0, 1] / nb, (S[0, 0] + S[1, 1]) / (2 * nb)
    rt, al = torch.hypot(hx, mxy), 0.5 * torch.atan2(2 * mxy, 2 * hx)
    ea, eb = torch.sqrt(2 * (tr + rt)), torch.sqrt(torch.clamp(2 * (tr - rt), min=0.0))
    a, p, q = 0.5 * L, 1 + math.sqrt(2.0), 1 - math.sqrt(2.0)
    rs = torch.clamp(r, min=float(1e-6 * L))
    u, v = (dx * al.cos() + dy * al.sin()) / rs, (dy * al.cos() - dx * al.sin()) / rs
    rb = ea * eb / torch.sqrt(eb * eb * u * u + ea * ea * v * v)
    rho = torch.minimum(rs * a / torch.maximum(rb, 1e-6 * L), 0.999999 * R)
    psi = a * ((rho / R) ** p - (rho / R) ** q) / ((a / R) ** p - (a / R) ** q) / rho
    inside = r < R
    phi = torch.where(inside, (R * R - r * r) / (R * R - a * a), torch.zeros_like(r))
    psi = torch.where(inside, psi, torch.zeros_like(r))
    kind = torch.zeros_like(x)
    kind[body], kind[outer] = 1.0, 2.0
    one = torch.ones_like(x)
    f = torch.stack([dx / L, dy / L, torch.log(r / L + 1e-6), torch.log(R / L) * one,
                     (kind == 1).double(), (kind == 2).double(), phi.clamp(0, 1), psi * dx / L,
                     psi * dy / L, eb / ea * one], 1)
    el = _t(k.inpoel.astype(np.int64) - 1)
    n = k.npoin
    e = torch.cat([el[:, [i, j]] for i in range(3) for j in range(3) if i != j])
    e = torch.unique(e[:, 0] * n + e[:, 1])
    src, dst = e // n, e % n
    ex, ey = x[dst] - x[src], y[dst] - y[src]
    ln = torch.hypot(ex, ey)
    ef = torch.stack([ex / ln, ey / ln, torch.log(ln / L)], 1)
    deg = torch.zeros(n, dtype=f.dtype, device=f.device).index_add_(0, src, torch.ones_like(ln))

    def forward(w):
        at = [0]

        def take(*shape):
            at[0] += math.prod(shape)
            return w[at[0] - math.prod(shape):at[0]].reshape(shape)

        W, b = take(64, 10), take(64)
        h = torch.relu(f @ W.T + b)
        for _ in range(4):
            A, B, C, c, Uw, ub = take(64, 64), take(64, 64), take(64, 3), take(64), take(64, 128), \
                take(64)
            z = torch.relu((h @ A.T)[src] + (h @ B.T)[dst] + ef @ C.T + c)
            agg = torch.zeros_like(h).index_add(0, src, z) / deg[:, None]
            h = h + torch.relu(torch.cat([h, agg], 1) @ Uw.T + ub)
        W, b = take(3, 64), take(3)
        return h @ W.T + b

    g = torch.stack([_t(gx), _t(gy)], 1)[:nb]
    M = torch.linalg.solve(S, D.T @ g).T
    return forward, kind, L, g.mean(0), M


def _exact_infer(c, seed):
    k = _mesh(c, seed)
    gx, gy = _rigid(k, np.random.default_rng(seed))
    forward, kind, L, t, M = _net64(k, gx, gy)
    with torch.no_grad():
        y = forward(_t(np.load(learned.DEFAULT_WEIGHTS)["weights"].astype(np.float64)))
        out = [t[q] * y[:, 0] + L * (M[q, 0] * y[:, 1] + M[q, 1] * y[:, 2]) for q in (0, 1)]
    node = _t(learned.boundary_of(k)[0].astype(np.int64) - 1)
    for o, g in zip(out, (gx, gy)):
        o[node] = _t(g)
    return tuple(o.cpu().numpy() for o in out)


def _exact_train(c, seed):
    k = _mesh(c, seed)
    zero = np.zeros(len(k.i_m) + len(k.ifm))
    forward, kind, L, _, _ = _net64(k, zero, zero)
    phi, px, py = (_t(v) for v in _targets(k, seed))
    w = _t(np.load(learned.DEFAULT_WEIGHTS)["weights"].astype(np.float64)).requires_grad_()
    free = kind == 0
    d = (forward(w) - torch.stack([phi, px / L, py / L], 1))[free]
    loss = (d * d).sum() / free.sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w.grad.cpu().numpy()}


def exact(case, seed):
    """run()'s outputs in plain 64-bit arithmetic.  A marched state has none: the plain form's
    ESTAB follows the direction of round-off, and the mixed form is held to the plain one."""
    kind = case["kind"]
    if kind == "bicg":
        return _exact_bicg(prepare(case, seed))
    if kind == "calcrhs":
        return _exact_rhs(prepare(case, seed))
    if kind == "infer":
        # 6 n edges x 64 doubles, several times over: up to about 600,000 nodes
        return _exact_infer(case, int(seed)) if case["nr"] * case["ntheta"] <= 1.2e6 else None
    if kind == "train":
        return _exact_train(case, int(seed))
    return None
