"""The calls of the design loop that are timed, over the sizes they are used at.

A pass is what a user's program does with objects that it keeps: one design
evaluation (initial state, checkpoints, objective with sensitivities, volume
constraint), one filter application with its chain rule, or one MMA update.
Inputs are float64 CUDA tensors in DMDA natural order.
"""
import math

import numpy as np
import torch

import topopt_in_petsc_transient_gb300 as tg

# Cantilever workloads of the benchmark: unit elements, E0 = 1, Emin = 1e-9,
# density 1 (1e-3 in the void), SIMP p = 3, Rayleigh damping beta = 1e-3 on
# the stiffness; time steps far below the element's wave transit time.
CANTILEVER = (1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)
# Default materials of TopOpt (Emax = 1e3, Rmax = 4.1667e-4): time steps of 1,
# so the step operator is dominated by its stiffness.
DEFAULTS = (1e-6, 1e3, 4.16666666667e-7, 4.16666666667e-4, 3.0, 1.0)
VOLFRAC = 0.12


def listed():
    def ev(name, nx, ny, nz, **kw):
        c = dict(name=name, kind="evaluate", nelx=nx, nely=ny, nelz=nz, nlvls=1, ncp=1, tsc=20, dt=0.01, objective=3,
                 mixed=True, material="cantilever", noise=0.02, load2=False, ti=1, basis=0)
        c.update(kw)
        return c

    def fl(name, nx, ny, nz, **kw):
        c = dict(name=name, kind="filter", nelx=nx, nely=ny, nelz=nz, filter=2, rmin=2.0, projection=True)
        c.update(kw)
        return c

    return [
        # the beam of the tests: launches and latency are all there is
        ev("eval_16x8x8", 16, 8, 8, nlvls=3, ncp=2, tsc=20),
        # the small benchmark cantilever on the plain FP64 path (100 steps)
        ev("eval_48x24x24_fp64", 48, 24, 24, nlvls=4, ncp=4, tsc=25, mixed=False),
        # an odd mesh (no coarser multigrid level), backward Euler, energy objective
        ev("eval_61x37x30_odd", 61, 37, 30, ncp=3, tsc=9, dt=0.02, objective=5, ti=0, noise=0.05),
        # the default TopOpt configuration: multigrid-preconditioned solves
        ev("eval_64x32x32_defaults", 64, 32, 32, nlvls=4, ncp=2, tsc=25, dt=1.0, objective=0, material="defaults",
           noise=0.05),
        # the mid-size benchmark cantilever, all 200 steps
        ev("eval_96x48x48", 96, 48, 48, nlvls=5, ncp=10, tsc=20, dt=0.005),
        # the large benchmark cantilever with its second load, two checkpoint blocks of its 400 steps
        ev("eval_192x96x96", 192, 96, 96, nlvls=6, ncp=2, tsc=20, dt=0.0025, load2=True),
        # reduced-order evaluation on the SOMMG basis
        ev("sommg_48x24x24", 48, 24, 24, nlvls=4, ncp=1, tsc=200, dt=0.005, basis=8),
        # PDE filter with projection and chain rule: a small mesh and the large benchmark mesh
        fl("pde_filter_48x24x24", 48, 24, 24),
        fl("pde_filter_192x96x96", 192, 96, 96),
        # density filter (-filter 1) at the mid-size mesh
        fl("density_filter_96x48x48", 96, 48, 48, filter=1, rmin=3.0),
        # MMA: a small and the large design vector
        dict(name="mma_27648", kind="mma", n=27648),
        dict(name="mma_1769472", kind="mma", n=1769472),
    ]


def _box(rng, most):
    """A beam-shaped mesh of at most `most` elements, its size spread over the logarithm."""
    nel = math.exp(rng.uniform(math.log(600.0), math.log(float(most))))
    ry, rz = rng.uniform(0.35, 0.7), rng.uniform(0.35, 0.7)
    nx = (nel / (ry * rz)) ** (1.0 / 3.0)
    return max(4, int(nx)), max(3, int(nx * ry)), max(3, int(nx * rz))


def draw(rng):
    kind = rng.choice(["evaluate"] * 5 + ["filter"] * 2 + ["mma"])
    if kind == "mma":
        return dict(kind="mma", n=int(math.exp(rng.uniform(math.log(500), math.log(1769472)))))
    if kind == "filter":
        t = rng.choice([2, 2, 1, 0])
        nx, ny, nz = _box(rng, 1500000 if t == 2 else 200000)
        return dict(kind="filter", nelx=nx, nely=ny, nelz=nz, filter=t,
                    rmin=round(rng.uniform(1.2, 3.0) if t == 2 else rng.uniform(2.1, 3.4), 3),
                    projection=rng.random() < 0.7)
    how = rng.choice(["mixed", "mixed", "mixed", "fp64", "defaults"])
    nx, ny, nz = _box(rng, {"mixed": 1200000, "fp64": 40000, "defaults": 60000}[how])
    nlvls = 1
    if how == "defaults":  # the multigrid levels need even element counts
        nlvls = 3
        nx, ny, nz = (max(8, v // 4 * 4) for v in (nx, ny, nz))
    nz += nz % 2  # the line load sits on the nodes at mid height
    nel = nx * ny * nz
    # as many steps as the large listed cantilever's work allows, at most 120
    steps = max(4, min(120, int((25e6 if how == "mixed" else 1.5e6) / nel)))
    ncp = rng.choice([c for c in (1, 2, 3, 4) if steps // c >= 2])
    dt = 1.0 if how == "defaults" else round(math.exp(rng.uniform(math.log(0.0025), math.log(0.02))), 5)
    return dict(kind="evaluate", nelx=nx, nely=ny, nelz=nz, nlvls=nlvls, ncp=ncp, tsc=max(2, steps // ncp), dt=dt,
                objective=rng.choice([0, 3, 3, 5]), mixed=how != "fp64",
                material="defaults" if how == "defaults" else "cantilever", noise=round(rng.uniform(0.0, 0.06), 3),
                load2=how == "mixed" and rng.random() < 0.3, ti=1, basis=0)


def _nel(c):
    return c["nelx"] * c["nely"] * c["nelz"] if "nelx" in c else c["n"]


def _uniform(n, seed, k, lo=0.0, hi=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(7919 * int(seed) + k)
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)


def _second_load(c, seed):
    """Node and phase of the second point load, from the seed."""
    r = np.random.default_rng(int(seed))
    nx, ny, nz = c["nelx"] + 1, c["nely"] + 1, c["nelz"] + 1
    i, j, k = int(r.integers(nx // 2, nx)), int(r.integers(0, ny)), int(r.integers(0, nz))
    return i + nx * (j + ny * k), float(r.uniform(0.0, 2.0 * math.pi))


def _inputs(c, seed):
    """The seeded inputs, the same for prepare() and exact()."""
    n = _nel(c)
    if c["kind"] == "evaluate":
        return dict(x=_uniform(n, seed, 1, VOLFRAC - c["noise"], VOLFRAC + c["noise"]))
    if c["kind"] == "filter":
        # a design in progress and sensitivities of one sign spread over magnitudes, as an objective's are
        return dict(x=_uniform(n, seed, 1, 0.02, 0.98), dfdx=-(_uniform(n, seed, 2) ** 4), dgdx=torch.full(
            (n,), 1.0 / n, dtype=torch.float64, device="cuda"))
    # an MMA update in the middle of an optimisation: two older designs and asymptotes around the current one
    x = _uniform(n, seed, 1, 0.05, 0.6)
    xo1 = (x + _uniform(n, seed, 2, -0.03, 0.03)).clamp(0.0, 1.0)
    xo2 = (xo1 + _uniform(n, seed, 3, -0.03, 0.03)).clamp(0.0, 1.0)
    return dict(x=x, xo1=xo1, xo2=xo2, low=xo1 - _uniform(n, seed, 4, 0.05, 0.3), upp=xo1 + _uniform(n, seed, 5, 0.05, 0.3),
                dfdx=-1e2 * _uniform(n, seed, 6) ** 4 / n,
                dgdx=torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda"))


def prepare(case, seed):
    c = case
    s = dict(case=c, **_inputs(c, seed))
    if c["kind"] == "evaluate":
        node, phase = _second_load(c, seed) if c["load2"] else (-1, 0.0)
        dflt = c["material"] == "defaults"
        s["physics"] = tg.LinearElasticity(
            c["nelx"], c["nely"], c["nelz"], nlvls=c["nlvls"], ncp=c["ncp"], tsc=c["tsc"],
            t1=c["dt"] * c["ncp"] * c["tsc"], ti=c["ti"], objective=c["objective"], mixed=c["mixed"],
            loadsignal=0 if dflt else 1, dalpha=1e-4 if dflt else 0.0, dbeta=1e-4 if dflt else 1e-3,
            load2_node=node, load2_phase=phase, reduction=c["basis"] > 0, basis=max(1, c["basis"]),
            omega0=_omega0(c))
        s["material"] = DEFAULTS if dflt else CANTILEVER
        s["dfdx"], s["dgdx"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
    elif c["kind"] == "filter":
        s["filter"] = tg.Filter(c["nelx"], c["nely"], c["nelz"], c["filter"], c["rmin"])
        s["xTilde"], s["xPhys"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
        s["df"], s["dg"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
    else:
        s["mma"] = tg.MMA(c["n"], 1, itr=10, xo1=s["xo1"], xo2=s["xo2"], U=s["upp"], L=s["low"])
        s["mma"].SetAsymptotes(0.1, 0.6, 1.05)
        s["gx"] = float(s["x"].mean()) - 0.3
        s["xnew"], s["xold"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
        s["xmin"], s["xmax"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
    torch.cuda.synchronize()  # the objects read the inputs on streams of their own
    return s


def _omega0(c):
    # half the first eigenfrequency of a 2:1:1 beam at this density (0.061 / nelx)
    return 0.03 / c["nelx"]


def run(s):
    c = s["case"]
    if c["kind"] == "evaluate":
        ph = s["physics"]
        ph.CompleteInitialState(s["x"], *s["material"])
        ph.GenerateCheckPoints()
        fx = ph.ComputeObjectiveSensitivities(s["dfdx"])
        gx = ph.VolumeConstraint(s["dgdx"], s["x"], VOLFRAC)
        return dict(fx=fx, dfdx=s["dfdx"], gx=gx, dgdx=s["dgdx"])
    if c["kind"] == "filter":
        f, beta, eta = s["filter"], 4.0, 0.3
        f.FilterProject(s["x"], s["xTilde"], s["xPhys"], c["projection"], beta, eta)
        # Gradients works in place: the sensitivities are handed over in buffers of their own
        s["df"].copy_(s["dfdx"])
        s["dg"].copy_(s["dgdx"])
        torch.cuda.current_stream().synchronize()  # the library's streams do not wait for torch's
        f.Gradients(s["x"], s["xTilde"], s["df"], 1, s["dg"], c["projection"], beta, eta)
        return dict(xTilde=s["xTilde"], xPhys=s["xPhys"], dfdx=s["df"], dgdx=s["dg"])
    s["xnew"].copy_(s["x"])
    s["xold"].copy_(s["x"])
    torch.cuda.current_stream().synchronize()
    m = s["mma"]
    m.SetOuterMovelimit(0.0, 1.0, 0.2, s["xnew"], s["xmin"], s["xmax"])
    m.Update(s["xnew"], s["dfdx"], [s["gx"]], s["dgdx"], s["xmin"], s["xmax"])
    ch = m.DesignChange(s["xnew"], s["xold"])
    return dict(x=s["xnew"], xmin=s["xmin"], xmax=s["xmax"], ch=ch)


def work(case):
    """Vectors that have to be read and written once a pass and the multiply-adds of one operator product each."""
    c = case
    n = _nel(c)
    if c["kind"] == "mma":
        return dict(bytes=8.0 * n * (9 + 6), flops=60.0 * n)
    nn = (c["nelx"] + 1) * (c["nely"] + 1) * (c["nelz"] + 1)
    if c["kind"] == "filter":
        if c["filter"] == 2:  # three Helmholtz solves: right-hand side, solution, one product
            return dict(bytes=8.0 * n * 8 + 3 * 16.0 * nn, flops=3 * 54.0 * nn)
        w = 2 * int(math.ceil(c["rmin"]) - 1) + 1
        return dict(bytes=8.0 * n * 9, flops=3 * 2.0 * w ** 3 * n)
    steps = c["ncp"] * c["tsc"]
    prod = 2.0 * (45 + 24 + 117) * n  # stiffness and mass of an element in its mode basis
    if c["basis"]:
        k = c["basis"]
        return dict(bytes=8.0 * 3 * nn * 6 * k, flops=k * (6 * prod + 6.0 * nn * k))
    sweeps = steps * (2 if c["ncp"] > 1 else 1) - (c["tsc"] if c["ncp"] > 1 else 0)
    # a forward step reads and writes a state (u, du, ddu); an adjoint step reads one and the adjoint triple, and
    # writes that; each solves once
    return dict(bytes=8.0 * 3 * nn * (6.0 * sweeps + 9.0 * steps) + 40.0 * n, flops=prod * 2.0 * (sweeps + steps))


# --- the same results in 64 bits from plain torch --------------------------------------------------------------------


def _hex8():
    """Stiffness (E = 1, nu = 0.3) and mass of the unit hex8 element, 2 x 2 x 2 Gauss points, DOF 3 L + c with the
    node L = ax + 2 ay + 4 az."""
    nu = 0.3
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[np.arange(3), np.arange(3)] += 2 * mu
    D[np.arange(3, 6), np.arange(3, 6)] = mu
    K, M = np.zeros((24, 24)), np.zeros((24, 24))
    p = 0.5 / math.sqrt(3.0)
    for q in range(8):
        xi = [0.5 + (p if (q >> a) & 1 else -p) for a in range(3)]
        N, G = np.zeros(8), np.zeros((8, 3))
        for L in range(8):
            f = [xi[a] if (L >> a) & 1 else 1 - xi[a] for a in range(3)]
            d = [1.0 if (L >> a) & 1 else -1.0 for a in range(3)]
            N[L] = f[0] * f[1] * f[2]
            G[L] = [d[0] * f[1] * f[2], f[0] * d[1] * f[2], f[0] * f[1] * d[2]]
        B, S = np.zeros((6, 24)), np.zeros((3, 24))
        for L in range(8):
            gx, gy, gz = G[L]
            B[:, 3 * L:3 * L + 3] = [[gx, 0, 0], [0, gy, 0], [0, 0, gz], [gy, gx, 0], [0, gz, gy], [gz, 0, gx]]
            S[:, 3 * L:3 * L + 3] = N[L] * np.eye(3)
        K += B.T @ D @ B / 8
        M += S.T @ S / 8
    return torch.tensor(K, device="cuda"), torch.tensor(M, device="cuda")


def _corners(c):
    """Node numbers [nel, 8] of every element, node L = ax + 2 ay + 4 az."""
    nx, ny, nz = c["nelx"] + 1, c["nely"] + 1, c["nelz"] + 1
    n = torch.arange(nx * ny * nz, device="cuda").view(nz, ny, nx)
    return torch.stack([n[(L >> 2):nz - 1 + (L >> 2), ((L >> 1) & 1):ny - 1 + ((L >> 1) & 1), (L & 1):nx - 1 + (L & 1)]
                        .reshape(-1) for L in range(8)], 1)


def _exact_evaluate(c, seed):
    nel = _nel(c)
    steps, dt = c["ncp"] * c["tsc"], c["dt"]
    if c["basis"] or c["material"] == "defaults" or nel * steps > 80e6:
        return None  # the basis has no plain counterpart; the others take too long
    x = _inputs(c, seed)["x"]
    Emin, Emax, Rmin, Rmax, pK, _ = CANTILEVER
    kf, dkf = Emin + x ** pK * (Emax - Emin), pK * x ** (pK - 1) * (Emax - Emin)
    mf, dmf = Rmin + x * (Rmax - Rmin), torch.full_like(x, Rmax - Rmin)
    al, be = 0.0, 1e-3
    nx, ny, nz = c["nelx"] + 1, c["nely"] + 1, c["nelz"] + 1
    nn = nx * ny * nz
    KE, ME = _hex8()
    corner = _corners(c)
    dofs = (3 * corner.unsqueeze(2) + torch.arange(3, device="cuda")).reshape(nel, 24)
    flat = dofs.reshape(-1)
    free = torch.ones(nz, ny, nx, 3, dtype=torch.float64, device="cuda")
    free[:, :, 0] = 0.0
    free = free.reshape(-1)

    def assemble(ye):
        return torch.zeros(3 * nn, dtype=torch.float64, device="cuda").index_add_(0, flat, ye.reshape(-1))

    def product(ck, cm, v):
        ve = v[dofs]
        return assemble((ve @ KE) * ck[:, None] + (ve @ ME) * cm[:, None])

    def mass(cm, v):
        return assemble((v[dofs] @ ME) * cm[:, None])

    if c["ti"] == 0:
        a = [0.0, 0.0, 1 / dt, 1 / dt, 0.0, 1 / dt ** 2]
    else:
        a = [-1.0, 0.0, 2 / dt, 4 / dt, 1.0, 4 / dt ** 2]
    sK, sM = 1 + a[2] * be, a[5] + a[2] * al
    one = torch.ones(nel, 24, dtype=torch.float64, device="cuda")

    def solver(ck, cm):
        dinv = 1.0 / assemble(one * torch.diagonal(KE) * ck[:, None] + one * torch.diagonal(ME) * cm[:, None])

        def solve(b, x0):
            b = b * free
            u = x0 * free
            r = b - free * product(ck, cm, u)
            bb = float(b @ b)
            if bb == 0.0:
                return torch.zeros_like(b)
            z = dinv * r * free
            p, rz = z.clone(), r @ z
            for it in range(2000):
                if it % 4 == 0 and float(r @ r) <= 1e-26 * bb:
                    break
                q = free * product(ck, cm, p)
                t = rz / (p @ q)
                u = u + t * p
                r = r - t * q
                z = dinv * r * free
                rz, old = r @ z, rz
                p = z + (rz / old) * p
            return u
        return solve

    solve, solve_mass = solver(sK * kf, sM * mf), solver(0 * kf, mf)
    load0 = torch.zeros(nz, ny, nx, 3, dtype=torch.float64, device="cuda")
    load0[c["nelz"] // 2, :, -1, 2] = 1.0
    load0[c["nelz"] // 2, 0, -1, 2] = load0[c["nelz"] // 2, -1, -1, 2] = 0.5
    load0 = load0.reshape(-1)
    node, phase = _second_load(c, seed) if c["load2"] else (-1, 0.0)

    def force(t):
        f = load0 * (math.sin(2 * math.pi * t) if t < 0.5 else 0.0) / (ny - 1)
        if node >= 0 and t < 0.5:
            f[3 * node + 2] += math.sin(2 * math.pi * t + phase) / (ny - 1)
        return f * free

    zero = torch.zeros(3 * nn, dtype=torch.float64, device="cuda")
    U, V, A = [zero], [zero], [solve_mass(force(0.0), zero)]
    for n in range(1, steps + 1):
        u, v, w = U[-1], V[-1], A[-1]
        cm = (sM * u + (a[3] - a[0] * al) * v + (a[4] - a[1] * al) * w)
        ck = be * (a[2] * u - a[0] * v - a[1] * w)
        b = force(n * dt) + (mass(mf, cm) + product(kf, 0 * mf, ck))
        un = solve(b, u + dt * v + 0.5 * dt * dt * w)
        du = un - u
        U.append(un)
        V.append(a[0] * v + a[1] * w + a[2] * du)
        A.append(-a[3] * v - a[4] * w + a[5] * du)

    obj = c["objective"]
    cnt = torch.zeros(nn, dtype=torch.float64, device="cuda").index_add_(
        0, corner.reshape(-1), torch.ones(8 * nel, dtype=torch.float64, device="cuda")).repeat_interleave(3)

    def energies(u, v):
        ue, ve = u[dofs], v[dofs]
        return ((ue @ KE) * ue).sum(1), ((ve @ ME) * ve).sum(1)

    def value(u, v):
        """Objective of a state, its derivative by the densities and by (u, v)."""
        if obj == 0:
            return 0.5 * dt * float(cnt @ (u * u)), 0.0, dt * cnt * u, zero
        k, m = energies(u, v)
        g = product(dt * kf, 0 * mf, u)
        if obj == 3:
            return 0.5 * dt * float(kf @ k), 0.5 * dt * dkf * k, g, zero
        return (0.5 * dt * float(kf @ k + mf @ m), 0.5 * dt * (dkf * k + dmf * m), g, mass(dt * mf, v))

    fx, df = 0.0, torch.zeros(nel, dtype=torch.float64, device="cuda")
    # reverse sweep: (gu, gv, ga) is the derivative of everything after step n by its state
    gu = gv = ga = zero
    lam = zero
    for n in range(steps, 0, -1):
        f, d, hu, hv = value(U[n], V[n])
        fx, df = fx + f, df + d
        gu, gv = gu + hu, gv + hv
        # v = .. + a2 u, w = .. + a5 u of the same step, then the solve
        lam = solve(gu + a[2] * gv + a[5] * ga, lam)
        u, v, w, un = U[n - 1], V[n - 1], A[n - 1], U[n]
        wm = sM * u + (a[3] - a[0] * al) * v + (a[4] - a[1] * al) * w - sM * un
        wk = be * (a[2] * u - a[0] * v - a[1] * w) - sK * un
        le = lam[dofs]
        df = df + dkf * ((le @ KE) * wk[dofs]).sum(1) + dmf * ((le @ ME) * wm[dofs]).sum(1)
        Kl, Ml = free * product(kf, 0 * mf, lam), free * mass(mf, lam)
        gu, gv, ga = (sM * Ml + be * a[2] * Kl - a[2] * gv - a[5] * ga,
                      (a[3] - a[0] * al) * Ml - be * a[0] * Kl + a[0] * gv - a[3] * ga,
                      (a[4] - a[1] * al) * Ml - be * a[1] * Kl + a[1] * gv - a[4] * ga)
    f, d, hu, hv = value(U[0], V[0])  # the state at rest: its displacement and velocity do not move
    fx, df = fx + f, df + d
    lam = solve_mass(ga, zero)
    df = df - dmf * ((lam[dofs] @ ME) * A[0][dofs]).sum(1)
    return dict(fx=fx, dfdx=df, gx=float(x.mean()) - VOLFRAC, dgdx=torch.full_like(x, 1.0 / nel))


def _axis(v, f):
    """The matrices f[0], f[1], f[2] applied along x, y, z of the node box."""
    v = torch.einsum("ai,kji->kja", f[0], v)
    v = torch.einsum("aj,kji->kai", f[1], v)
    return torch.einsum("ak,kji->aji", f[2], v)


def _exact_filter(c, seed):
    s = _inputs(c, seed)
    ex, ey, ez = c["nelx"], c["nely"], c["nelz"]
    if c["filter"] == 2:
        R = c["rmin"] / 2.0 / math.sqrt(3.0)
        Q, W = [], []
        for n in (ex + 1, ey + 1, ez + 1):  # eigenvectors of the 1-D stiffness by the 1-D mass
            K, M = np.zeros((n, n)), np.zeros((n, n))
            for e in range(n - 1):
                K[e:e + 2, e:e + 2] += [[1, -1], [-1, 1]]
                M[e:e + 2, e:e + 2] += np.array([[2, 1], [1, 2]]) / 6.0
            Li = np.linalg.inv(np.linalg.cholesky(M))
            w, q = np.linalg.eigh(Li @ K @ Li.T)
            Q.append(torch.tensor(Li.T @ q, device="cuda"))
            W.append(torch.tensor(w, device="cuda"))
        den = R * R * (W[2][:, None, None] + W[1][None, :, None] + W[0][None, None, :]) + 1.0
        corner = _corners(c).reshape(-1)

        def smooth(v):
            rhs = torch.zeros(den.numel(), dtype=torch.float64, device="cuda").index_add_(
                0, corner, (0.125 * v).repeat_interleave(8)).view_as(den)
            u = _axis(_axis(rhs, [q.T for q in Q]) / den, Q).reshape(-1)
            return 0.125 * u[corner].view(-1, 8).sum(1)

        back = smooth
        xt = smooth(s["x"]).clamp(0.0, 1.0)
    else:
        R = c["rmin"]
        w = int(math.ceil(R)) - 1

        def H(v):
            v = v.view(ez, ey, ex)
            if w <= 1:
                return v.reshape(-1).clone()
            out = torch.zeros_like(v)
            for dz in range(-w, w + 1):
                for dy in range(-w, w + 1):
                    for dx in range(-w, w + 1):
                        q = R - math.sqrt(dx * dx + dy * dy + dz * dz)
                        if q <= 0 or abs(dz) >= ez or abs(dy) >= ey or abs(dx) >= ex:
                            continue
                        lo = [max(0, -d) for d in (dz, dy, dx)]
                        hi = [n - max(0, d) for n, d in zip((ez, ey, ex), (dz, dy, dx))]
                        out[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] += q * v[
                            lo[0] + dz:hi[0] + dz, lo[1] + dy:hi[1] + dy, lo[2] + dx:hi[2] + dx]
            return out.reshape(-1)
        hs = H(torch.ones_like(s["x"])) if w > 1 else torch.ones_like(s["x"])
        xt = H(s["x"]) / hs if c["filter"] == 1 else s["x"]

        def back(v):
            return H(v / hs)
    beta, eta = 4.0, 0.3
    den1 = math.tanh(beta * eta) + math.tanh(beta * (1 - eta))
    xp, df, dg = xt, s["dfdx"], s["dgdx"]
    if c["projection"]:
        t = torch.tanh(beta * (xt - eta))
        xp = (math.tanh(beta * eta) + t) / den1
        df, dg = df * (beta * (1 - t * t) / den1), dg * (beta * (1 - t * t) / den1)
    if c["filter"] == 0:  # the sensitivity filter leaves the constraint's alone
        df = H(df * s["x"]) / hs / s["x"]
    else:
        df, dg = back(df), back(dg)
    return dict(xTilde=xt, xPhys=xp, dfdx=df, dgdx=dg)


def _exact_mma(c, seed):
    s = _inputs(c, seed)
    x, n = s["x"], c["n"]
    lo, hi = (x - 0.2).clamp(min=0.0), (x + 0.2).clamp(max=1.0)
    h = (x - s["xo1"]) * (s["xo1"] - s["xo2"])
    g = torch.where(h < 0, torch.full_like(x, 0.6), torch.where(h > 0, torch.full_like(x, 1.05), torch.ones_like(x)))
    xmi = (hi - lo).clamp(min=1e-5)
    L = torch.minimum(torch.maximum(x - g * (s["xo1"] - s["low"]), x - 10 * xmi), x - 0.01 * xmi)
    U = torch.minimum(torch.maximum(x + g * (s["upp"] - s["xo1"]), x + 0.01 * xmi), x + 10 * xmi)
    al, be = torch.maximum(lo, 0.9 * L + 0.1 * x), torch.minimum(hi, 0.9 * U + 0.1 * x)
    df, dg = s["dfdx"], s["dgdx"]
    base = 0.001 * df.abs() + 0.5e-6 / (U - L)
    p0, q0 = (U - x) ** 2 * (df.clamp(min=0) + base), (x - L) ** 2 * ((-df).clamp(min=0) + base)
    p1, q1 = (U - x) ** 2 * dg.clamp(min=0), (x - L) ** 2 * (-dg).clamp(min=0)
    b = float((p1 / (U - x) + q1 / (x - L)).sum()) - (float(x.mean()) - 0.3)
    cc = 1000.0
    lam, mu, epsi, err = cc / 2, 1.0, 1.0, 1.0

    def at(l):
        p, q = p0 + l * p1, q0 + l * q1
        raw = (p.sqrt() * L + q.sqrt() * U) / (p.sqrt() + q.sqrt())
        v = torch.minimum(torch.maximum(raw, al), be)
        return p, q, raw, v, float((p1 / (U - v) + q1 / (v - L)).sum()) - b - max(0.0, l - cc)

    p, q, raw, v, grad = at(lam)
    while epsi > 1e-9 * math.sqrt(1 + n):
        for _ in range(100):
            if not err > 0.9 * epsi:
                break
            pq = p1 / (U - v) ** 2 - q1 / (v - L) ** 2
            d2 = -1.0 / (2 * p / (U - v) ** 3 + 2 * q / (v - L) ** 3)
            d2 = torch.where((raw < al) | (raw > be), torch.zeros_like(d2), d2)
            H = float((pq * d2 * pq).sum()) + (-1.0 if lam > cc else 0.0) - mu / lam
            corr = 1e-4 * H
            H += -1e-7 if -corr < 1e-7 else corr
            st = (-grad - epsi / lam) / H
            sm = -mu + epsi / lam - st * mu / lam
            th = 1.0 / max(1.005, -1.01 * st / lam, -1.01 * sm / mu)
            lam, mu = max(0.0, lam + th * st), mu + th * sm
            p, q, raw, v, grad = at(lam)
            err = max(abs(grad + mu), abs(mu * lam - epsi))
        epsi *= 0.1
    return dict(x=v, xmin=lo, xmax=hi, ch=float((v - x).abs().max()))


def exact(case, seed):
    return {"evaluate": _exact_evaluate, "filter": _exact_filter, "mma": _exact_mma}[case["kind"]](case, seed)
