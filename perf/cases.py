"""The work this framework is used for, as cases that can be timed and compared: velocity solves, the
matrix-equation solve, operator application, column thermodynamics, the ice-thickness step, and the
learned start's network in both directions, from the smallest calls to the largest meshes of this
repository's own workloads.

Every case calls the public Python entry points with host arrays, as a host model's program does;
meshes come from the package's generators (built once per size and kept), the ice state from the seed.
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__ as _entry

pkg = _entry.load_package()
geo = pkg.geometry


# ---- meshes: one per kind and size, kept for the life of the process -----------------------------
@functools.lru_cache(maxsize=None)
def _dome(nV):
    return geo.dome_case(res_scale=math.sqrt(8492.0 / nV))


@functools.lru_cache(maxsize=None)
def _channel(nV, nz):
    return geo.channel_case(res_scale=math.sqrt(58243.0 / nV), nz=nz)


@functools.lru_cache(maxsize=None)
def _thermo(nV, nz):
    return geo.thermo_case(nV=nV, nz=nz)


@functools.lru_cache(maxsize=None)
def _thickness(nV):
    L = 800e3
    mesh, fields, params = geo.thickness_case(L=L, res=L / 2 ** math.floor(0.5 * math.log2(nV)) * 1.001)
    return mesh, fields, params, pkg.mesh.voronoi_geometry(mesh)


@functools.lru_cache(maxsize=None)
def _graph(nTri):
    """Triangle adjacency (-1: none) of a channel mesh, the triangles along a Z-order curve as the
    library numbers them."""
    mesh = _channel(nTri // 2, 12)[0]
    gc = np.asarray(mesh.TriGC)
    q = ((gc - gc.min(0)) / np.ptp(gc) * 4095.0).astype(np.int64)
    code = np.zeros(mesh.nTri, np.int64)
    for bit in range(12):
        code |= (((q[:, 0] >> bit) & 1) << (2 * bit)) | (((q[:, 1] >> bit) & 1) << (2 * bit + 1))
    order = np.argsort(code, kind="stable")
    new = np.empty(mesh.nTri, np.int64)
    new[order] = np.arange(mesh.nTri)
    nbr = np.asarray(mesh.TriC, np.int64)[order] - 1
    return np.ascontiguousarray(np.where(nbr >= 0, new[nbr], -1).astype(np.int32))


# ---- seeded inputs -------------------------------------------------------------------------------
def _dome_ice(mesh, base, seed):
    """The SSA dome with another height, a rough surface of a few per cent and a log-normal friction."""
    rng = np.random.default_rng(seed)
    x, y = mesh.V[:, 0], mesh.V[:, 1]
    Hi = base["Hi"] * rng.uniform(0.97, 1.03) * (1.0 + 0.02 * geo.smooth_field(x, y, 80e3, seed + 1, n_modes=24))
    beta = base["beta_sq"] * np.exp(0.3 * geo.smooth_field(x, y, 60e3, seed + 2, n_modes=24))
    return dict(base, Hi=np.ascontiguousarray(Hi), Hs=np.ascontiguousarray(geo.surface_elevation(Hi, base["Hb"], base["SL"])),
                mask_grounded_ice=np.ascontiguousarray((Hi > 0).astype(np.int32)), beta_sq=np.ascontiguousarray(beta))


def _channel_ice(mesh, base, seed):
    """The MISMIP+-shaped channel with another thickness, flow factor and friction."""
    rng = np.random.default_rng(seed)
    H, A = rng.uniform(240.0, 260.0), 2e-17 * rng.uniform(0.9, 1.1)
    Hb, SL = base["Hb"], base["SL"]
    Hi = np.full(mesh.nV, H)
    taf = geo.thickness_above_flotation(Hi, Hb, SL)
    effp = np.maximum(0.0, geo.ICE_DENSITY * geo.GRAV * Hi - geo.SEAWATER_DENSITY * geo.GRAV * np.maximum(0.0, SL - Hb))
    return dict(base, Hi=Hi, Hs=np.ascontiguousarray(geo.surface_elevation(Hi, Hb, SL)),
                A_flow=np.asfortranarray(np.full((mesh.nV, mesh.nz), A)),
                fraction_gr_b=geo.grounded_fraction_b_vertex(mesh, taf, nsub=4),
                mask_grounded_ice=np.ascontiguousarray((taf > 0).astype(np.int32)),
                effective_pressure=np.ascontiguousarray(effp),
                beta_sq=np.full(mesh.nV, 1e4 * rng.uniform(0.8, 1.2)))


def _thermo_fields(mesh, base, seed):
    """The column fields with other temperatures, heating and vertical velocities."""
    rng = np.random.default_rng(seed)
    f = dict(base)
    zeta, n = mesh.zeta[None, :], mesh.nV
    T = base["Ti"] - rng.uniform(0.0, 3.0, (n, 1)) * np.sin(np.pi * zeta)
    f["Ti"] = np.asfortranarray(T)
    f["w_3D"] = np.asfortranarray(base["w_3D"] * rng.uniform(0.8, 1.2))
    f["internal_heating"] = np.asfortranarray(base["internal_heating"] * rng.uniform(0.5, 1.5, (n, 1)))
    f["geothermal_heat_flux"] = base["geothermal_heat_flux"] * rng.uniform(0.9, 1.1, n)
    return f


def _thickness_fields(mesh, base, seed):
    """The thickness step's fields with another thickness, flow and mass balance."""
    rng = np.random.default_rng(seed)
    f = dict(base)
    f["Hi"] = base["Hi"] * rng.uniform(0.98, 1.02, mesh.nV)
    turn = rng.uniform(-0.2, 0.2)
    u, v = base["u_vav_b"], base["v_vav_b"]
    s = rng.uniform(0.9, 1.1, mesh.nTri)
    f["u_vav_b"], f["v_vav_b"] = s * (u * math.cos(turn) - v * math.sin(turn)), s * (u * math.sin(turn) + v * math.cos(turn))
    f["SMB"] = base["SMB"] + rng.normal(0.0, 0.05, mesh.nV)
    f["dHi_dt"] = 0.01 * rng.standard_normal(mesh.nV)
    return f


def _matrix(n, seed):
    """One implicit step of advection and diffusion with log-normal conductivities on a grid of about
    n unknowns (five entries a row, not symmetric): the kind of system a host model hands to the
    matrix-equation solve.  Returns CSR arrays (0-based) and a right-hand side."""
    rng = np.random.default_rng(seed)
    nx = int(math.sqrt(n))
    ny = n // nx
    i = np.arange(nx * ny).reshape(ny, nx)
    K = np.exp(rng.normal(0.0, 0.5, (ny, nx)))
    rows, cols, vals = [], [], []
    diag = np.ones((ny, nx))
    for dy, dx, adv in ((0, 1, -0.6), (0, -1, 0.6), (1, 0, -0.3), (-1, 0, 0.3)):
        ys = slice(max(0, -dy), ny - max(0, dy))
        xs = slice(max(0, -dx), nx - max(0, dx))
        yt = slice(max(0, dy), ny - max(0, -dy))
        xt = slice(max(0, dx), nx - max(0, -dx))
        c = 20.0 * 0.5 * (K[ys, xs] + K[yt, xt])
        rows.append(i[ys, xs].ravel())
        cols.append(i[yt, xt].ravel())
        vals.append((-(c + adv)).ravel())
        diag[ys, xs] += c
    rows.append(i.ravel())
    cols.append(i.ravel())
    vals.append(diag.ravel())
    rows, cols, vals = (np.concatenate(a) for a in (rows, cols, vals))
    order = np.lexsort((cols, rows))
    ptr = np.zeros(nx * ny + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=nx * ny), out=ptr[1:])
    return ptr, cols[order].astype(np.int32), np.ascontiguousarray(vals[order]), rng.standard_normal(nx * ny)


#: The network: 16 features, width 64, four layers, 3 outputs, as one flat vector in this order.
_LAYOUT = ([("We", (64, 16)), ("be", (64,))]
           + [(k + str(l), s) for l in range(4) for k, s in (("W1", (64, 128)), ("b1", (64,)), ("W2", (64, 64)), ("b2", (64,)))]
           + [("Wd", (3, 64)), ("bd", (3,))])


def _network(n, nbr, seed):
    rng = np.random.default_rng(seed)
    p = []
    for name, shape in _LAYOUT:
        gain = 0.5 if name.startswith("W2") else 1.4
        p.append(rng.uniform(-1.0, 1.0, shape) * (gain * math.sqrt(3.0 / shape[-1]) if name[0] == "W" else 0.05))
    x = rng.standard_normal((n, 16)).astype(np.float32)
    x[:, 13] = rng.random(n) < 0.9
    w = x[:, 13] / max(1.0, x[:, 13].sum())
    target = rng.standard_normal((n, 3)).astype(np.float32) * 0.5
    return np.concatenate([a.ravel() for a in p]).astype(np.float32), x, target, w.astype(np.float32)


# ---- the cases -----------------------------------------------------------------------------------
def listed():
    return [
        # The smallest velocity call: a coarse dome in a model's test or spin-up, called with host arrays
        # every time step; launches and host work count.
        {"name": "ssa_dome_0.7k", "kind": "ssa", "nV": 741},
        # The radially symmetric SSA dome at its full 8,492 vertices, plain FP64, through solve_SSA.
        {"name": "ssa_dome_8k", "kind": "ssa", "nV": 8492},
        # The DIVA channel (58,243 vertices) with the fast solver: double-word Krylov inside the inexact Picard
        # iteration; upload of the ice state, resident solve, download -- one velocity update of a time step.
        {"name": "diva_channel_58k_pair", "kind": "diva_fast", "nV": 58243, "nz": 12},
        # Plain FP64 DIVA through solve_DIVA, the drop-in call with 3-D velocities back, on a coarser channel.
        {"name": "diva_channel_7k_fp64", "kind": "diva", "nV": 7000, "nz": 12},
        # The matrix-equation solve on a caller's CSR matrix.
        {"name": "csr_solve_60k", "kind": "csr", "n": 60000},
        # A host model's operator application: d/dx of a 3-D field from vertices to triangles.
        {"name": "ddx_a_b_3D_8k", "kind": "apply", "nV": 8492, "op": "DDX_A_B"},
        # Column thermodynamics on a caller's own columns, a small domain (12 layers).
        {"name": "thermo_columns_2k", "kind": "columns", "nV": 2000, "nz": 12, "stiff": 0.2},
        # The batched column workload, 200,000 columns of 30 layers: fields up, a coupling interval of ten
        # steps on the device, temperature back.
        {"name": "thermo_mesh_200k", "kind": "heat", "nV": 200000, "nz": 30, "steps": 10},
        # Ice thickness: one semi-implicit step of a large mesh, and one explicit step of a small one.
        {"name": "thickness_semi_260k", "kind": "thickness", "nV": 262144, "method": 2},
        {"name": "thickness_explicit_16k", "kind": "thickness", "nV": 16384, "method": 1},
        # The learned start's network: a prediction for the channel's 115k triangles, and the loss and
        # gradient of one training member on a 30,000-vertex mesh.
        {"name": "gnn_forward_115k", "kind": "gnn", "nTri": 115000, "train": False},
        {"name": "gnn_grad_60k", "kind": "gnn", "nTri": 60000, "train": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ssa", "ssa", "diva", "diva_fast", "csr", "apply", "columns", "heat", "thickness", "gnn", "gnn"])
    if kind == "ssa":
        return {"kind": kind, "nV": _log(rng, 500, 9000)}
    if kind in ("diva", "diva_fast"):
        return {"kind": kind, "nV": _log(rng, 1200, 7000 if kind == "diva" else 58000), "nz": rng.choice([7, 12, 15])}
    if kind == "csr":
        return {"kind": kind, "n": _log(rng, 900, 100000)}
    if kind == "apply":
        return {"kind": kind, "nV": _log(rng, 500, 30000),
                "op": rng.choice(["MAP_A_B", "DDX_A_B", "DDY_A_B", "MAP_B_A", "DDX_B_A", "DDY_B_A"])}
    if kind == "columns":
        return {"kind": kind, "nV": _log(rng, 503, 40000), "nz": rng.choice([5, 12, 13, 30, 41]), "stiff": rng.choice([0.0, 0.03])}
    if kind == "heat":
        return {"kind": kind, "nV": _log(rng, 2000, 60000), "nz": rng.choice([12, 23, 30]), "steps": rng.randint(1, 10)}
    if kind == "thickness":
        return {"kind": kind, "nV": 4 ** rng.randint(5, 9), "method": rng.choice([1, 2]), "dt": round(rng.uniform(0.2, 2.0), 3)}
    return {"kind": kind, "nTri": _log(rng, 1000, 200000), "train": rng.choice([True, False])}


def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k}
    if k in ("ssa", "diva", "diva_fast"):
        mesh, base, params = _dome(case["nV"]) if k == "ssa" else _channel(case["nV"], case["nz"])
        st["ice"] = (_dome_ice if k == "ssa" else _channel_ice)(mesh, base, seed)
        # the benchmark's tolerances: Picard 1e-4 (200 iterations at most), BiCGStab 1e-8
        st["params"] = pkg.abi.SolverParams.from_buffer_copy(params)
        st["params"].visc_it_nit = 200
        if k == "diva_fast":
            st["params"].precision = pkg.abi.PREC_FP32_PAIR
            st["params"].krylov_forcing = 0.1
        st["solver"] = pkg.VelocitySolver(mesh)
    elif k == "csr":
        ptr, ind, val, b = _matrix(case["n"], seed)
        st["A"] = pkg.CSR(len(b), len(b), ptr, ind, val, index_base=0)
        st["b"], st["x0"] = b, np.zeros(len(b))
        st["solver"] = pkg.VelocitySolver(_dome(741)[0])
    elif k == "apply":
        mesh = _dome(case["nV"])[0]
        n = mesh.nTri if "_B_A" in case["op"] else mesh.nV
        st["op"], st["solver"] = case["op"], pkg.VelocitySolver(mesh)
        st["x"] = np.asfortranarray(np.random.default_rng(seed).standard_normal((n, mesh.nz)))
    elif k == "columns":
        st["zeta"], st["cols"] = geo.random_columns(case["nV"], case["nz"], seed=seed, stiff_frac=case["stiff"], stiffness=3000.0)
        st["params"], st["solver"] = pkg.abi.default_thermo_params(dt=5.0), pkg.ColumnSolver()
    elif k == "heat":
        mesh, base, st["params"] = _thermo(case["nV"], case["nz"])
        st["fields"], st["steps"], st["solver"] = _thermo_fields(mesh, base, seed), case["steps"], pkg.VelocitySolver(mesh)
    elif k == "thickness":
        mesh, base, _, (A, Cw) = _thickness(case["nV"])
        st["fields"], st["dt"] = _thickness_fields(mesh, base, seed), case.get("dt", 1.0)
        st["params"] = pkg.abi.ThicknessParams.from_buffer_copy(_thickness(case["nV"])[2])
        st["params"].choice_ice_integration_method = case["method"]
        st["solver"] = pkg.VelocitySolver(mesh)
        st["solver"].voronoi_upload(A, Cw)
    else:
        st["nbr"] = _graph(case["nTri"])
        p, st["x"], st["target"], st["w"] = _network(len(st["nbr"]), st["nbr"], seed)
        st["train"], st["solver"] = case["train"], pkg.ColumnSolver()
        st["net"] = pkg.LearnedStart(st["solver"])
        st["net"].set_params(p)
    return st


def run(st):
    k, s = st["kind"], st["solver"]
    if k == "ssa":
        SSA = pkg.new_ssa_state(s.mesh.nTri)
        s.solve_SSA(st["ice"], SSA, st["params"])
        return SSA
    if k == "diva":
        DIVA = pkg.new_diva_state(s.mesh.nTri, s.mesh.nz)
        s.solve_DIVA(st["ice"], DIVA, st["params"])
        return DIVA
    if k == "diva_fast":
        s.ice_upload(st["ice"])
        s.solve_resident(st["params"], diva=True, cold_start=True)
        return s.velocity_download()
    if k == "csr":
        return s.solve_matrix_equation_CSR_PETSc(st["A"], st["b"], st["x0"], 1e-10, 0.0)[0]
    if k == "apply":
        return s.apply(st["op"], st["x"])
    if k == "columns":
        return s.thermo_step(st["params"], st["zeta"], st["cols"])
    if k == "heat":
        s.heat_upload(st["fields"])
        n, _ = s.heat_step_resident(st["params"], st["steps"])
        return s.heat_download(), n
    if k == "thickness":
        out = s.calc_dHi_dt(st["params"], st["fields"], st["dt"])
        # of the semi-implicit scheme AMB holds only what clipping H < 0 removed: the Krylov error's sign, no more
        names = ("dHi_dt", "Hi_tplusdt", "divQ", "dt") + (("AMB",) if st["params"].choice_ice_integration_method == 1 else ())
        return {name: out[name] for name in names}
    if st["train"]:
        return st["net"].loss_grad(st["nbr"], st["x"], st["target"], st["w"])
    return st["net"].forward(st["nbr"], st["x"])


def work(case):
    """Inputs read once and outputs written once.  For the iterative solves the operations of a nominal
    iteration count (Picard x Krylov as this repository's benchmark counts them) are in flops: per
    Krylov iteration two products with about 13 2x2 blocks a triangle and some 20 vector operations."""
    k = case["kind"]
    if k in ("ssa", "diva", "diva_fast"):
        nV, nT, nz = case["nV"], 2 * case["nV"], case.get("nz", 12)
        its = {"ssa": 2500, "diva": 12000, "diva_fast": 4000}[k]
        return {"bytes": 8.0 * (nV * (nz + 6) + 3 * nT + (3 * nz * nT + 6 * nT if k == "diva" else 0)),
                "flops": float(its) * nT * (2 * 13 * 8 + 40)}
    if k == "csr":
        return {"bytes": 12.0 * 5 * case["n"] + 28.0 * case["n"], "flops": 60.0 * case["n"] * (2 * 10 + 20)}
    if k == "apply":
        return {"bytes": 8.0 * 12 * 3 * case["nV"] + 12.0 * 13 * case["nV"], "flops": 2.0 * 12 * 13 * case["nV"]}
    if k == "columns":
        return {"bytes": 8.0 * case["nV"] * (12 * case["nz"] + 7), "flops": 120.0 * case["nV"] * case["nz"]}
    if k == "heat":
        nV, nz, st = case["nV"], case["nz"], case["steps"]
        return {"bytes": 8.0 * nV * (6 * nz + 4 * nz + 24) + st * 8.0 * nV * (8 * nz + 19), "flops": 120.0 * st * nV * nz}
    if k == "thickness":
        nV = case["nV"]
        return {"bytes": nV * (8.0 * (14 + 4 + 4) + 7 * 28.0), "flops": nV * (7 * 12.0 + (9 * 70.0 if case["method"] == 2 else 0.0))}
    n = case["nTri"]
    fwd = n * (2.0 * (16 * 64 + 4 * (128 * 64 + 64 * 64) + 3 * 64))
    return {"bytes": n * (4.0 * 16 + 12 + 12 + (16 if case["train"] else 0)), "flops": fwd * (3 if case["train"] else 1)}


# ---- what the outputs are in 64 bits, by plain numpy and torch ----------------------------------
def exact(case, seed):
    """None for the velocity solves, the operators and the mesh-level heat equation: they need the mesh
    discretisation and thousands of sparse iterations, minutes in plain torch."""
    k = case["kind"]
    if k == "csr":
        ptr, ind, val, b = _matrix(case["n"], seed)
        return _solve(ptr, ind, val, b)
    if k == "thickness":
        return _exact_thickness(case, seed)
    if k == "columns":
        return _exact_columns(case, seed)
    if k == "gnn":
        return _exact_network(case, seed)
    return None


def _solve(ptr, ind, val, b, x=None):
    """BiCGStab with Jacobi scaling, restarted from the true residual until that stops falling."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(np.asarray(a), device=dev)  # noqa: E731
    A = torch.sparse_csr_tensor(t(ptr).long(), t(ind).long(), t(val), size=(len(b), len(b)))
    row = np.repeat(np.arange(len(b)), np.diff(ptr))
    d = np.zeros(len(b))
    d[row[ind == row]] = val[ind == row]
    dinv, b = t(1.0 / d), t(b)
    x = torch.zeros_like(b) if x is None else t(x)
    mul = lambda y: dinv * (A @ y.unsqueeze(1)).squeeze(1)  # noqa: E731
    db, best = dinv * b, math.inf
    for _ in range(6):
        r = db - mul(x)
        norm = float(r.norm())
        if norm >= 0.5 * best or norm <= 1e-16 * float(db.norm()):
            break
        best, rh, p, e = norm, r.clone(), r.clone(), torch.zeros_like(x)
        rho = torch.dot(rh, r)
        for _ in range(2000):
            v = mul(p)
            a = rho / torch.dot(rh, v)
            s = r - a * v
            q = mul(s)
            w = torch.dot(q, s) / torch.dot(q, q)
            e = e + a * p + w * s
            r = s - w * q
            if float(r.norm()) <= 1e-9 * norm:
                break
            new = torch.dot(rh, r)
            p = r + (new / rho) * (a / w) * (p - w * v)
            rho = new
        x = x + e
    return x.cpu().numpy()


def _exact_thickness(case, seed):
    mesh, base, p, (A, Cw) = _thickness(case["nV"])
    f, dt = _thickness_fields(mesh, base, seed), float(case.get("dt", 1.0))
    nV, C, nC, VBI = mesh.nV, np.asarray(mesh.C, np.int64) - 1, np.asarray(mesh.nC), np.asarray(mesh.VBI)
    live = np.arange(mesh.nC_mem)[None, :] < nC[:, None]
    i = np.broadcast_to(np.arange(nV)[:, None], live.shape)[live]
    j = C[live]
    T = np.asarray(mesh.Tri, np.int64) - 1
    ends = np.concatenate([T[:, [0, 1]], T[:, [1, 2]], T[:, [2, 0]]])
    key = ends.min(1) * nV + ends.max(1)
    tri = np.tile(np.arange(mesh.nTri), 3)
    edges, inv, cnt = np.unique(key, return_inverse=True, return_counts=True)
    um = [np.bincount(inv.ravel(), weights=f[c][tri], minlength=len(edges)) / cnt for c in ("u_vav_b", "v_vav_b")]
    e = np.searchsorted(edges, np.minimum(i, j) * nV + np.maximum(i, j))
    V = np.asarray(mesh.V)
    D = V[j] - V[i]
    un = (um[0][e] * D[:, 0] + um[1][e] * D[:, 1]) / np.hypot(D[:, 0], D[:, 1])
    fm, Hi, Hb, SL = f["fraction_margin"], f["Hi"], f["Hb"], f["SL"]
    out = np.where((un > 0) & (fm[i] >= 1.0), Cw[live] * un / A[i], 0.0)
    off = np.where((un < 0) & (fm[j] >= 1.0), Cw[live] * un / A[i], 0.0)
    diag = np.bincount(i, weights=out, minlength=nV)
    divQ = diag * Hi + np.bincount(i, weights=off * Hi[j], minlength=nV)
    mb = fm * (f["SMB"] + f["BMB"] - f["dHi_dt_target"])
    noice, pres = f["mask_noice"] > 0, f["BC_prescr_mask"] == 1
    ratio = geo.ICE_DENSITY / geo.SEAWATER_DENSITY
    surface = lambda H: H + np.maximum(SL - ratio * H, Hb)  # noqa: E731
    side = np.select([(VBI == 1) | (VBI == 2), (VBI == 3) | (VBI == 4), (VBI == 5) | (VBI == 6), VBI >= 7],
                     [p.BC_H_north, p.BC_H_east, p.BC_H_south, p.BC_H_west], -1)
    inner = (VBI[j] == 0) & ~noice[j]
    nint = np.bincount(i, weights=inner, minlength=nV)

    def border(H):
        Hs = surface(H)
        H = H.copy()
        for k in (0, 1):
            tot = Hs.copy()
            mean = np.bincount(i, weights=tot[j] * (inner if k == 0 else 1.0), minlength=nV) / np.maximum(nint if k == 0 else nC, 1)
            at = (side == 1) & ((nint > 0) == (k == 0))
            Hs[at] = np.maximum(Hb[at], mean[at])
            fl = np.maximum(0.0, (SL - Hb) / ratio)
            new = np.where(Hs > Hb + fl, Hs - Hb, np.minimum(fl, (Hs - SL) / (1.0 - ratio)))
            H[at] = new[at]
            H[side == 0] = 0.0
        return H

    r = -divQ + mb + f["LMB"]
    thin = (Hi > p.Hi_min) & (r < 0)
    limit = min(p.dt_ice_max, float(np.min(Hi[thin] / 1e-9))) if thin.any() else p.dt_ice_max
    dte = min(dt, max(p.dt_ice_min, limit))
    H = border(np.maximum(0.0, Hi + r * dte))
    H[pres] = np.maximum(0.0, f["BC_prescr_Hi"][pres])
    H[noice] = 0.0
    if case["method"] == 1:
        rate = (H - Hi) / dte
        Hn = np.maximum(H, 0.0)
        return {"dHi_dt": (Hn - Hi) / dte, "Hi_tplusdt": Hn, "divQ": divQ, "AMB": rate - r + (Hn - Hi) / dte - rate, "dt": dte}
    H = border(H)
    fs = p.dHi_semiimplicit_fs
    b = Hi - dt * (1.0 - fs) * divQ + np.maximum(-Hi, dt * (mb + f["LMB"]))
    d, o = 1.0 + dt * fs * diag, dt * fs * off
    for at, val in ((VBI > 0, H), (pres, f["BC_prescr_Hi"]), (noice, np.zeros(nV))):
        b = np.where(at, val, b)
        d = np.where(at, 1.0, d)
        o = np.where(at[i], 0.0, o)
    x = b / d
    for _ in range(400):   # Jacobi: the rows are diagonally dominant for these time steps
        new = (b - np.bincount(i, weights=o * x[j], minlength=nV)) / d
        done = np.abs(new - x).max() <= 1e-13 * np.abs(new).max()
        x = new
        if done:
            break
    Hn = np.maximum(x, 0.0)
    return {"dHi_dt": (Hn - Hi) / dt, "Hi_tplusdt": Hn, "divQ": divQ, "dt": dt}


def _exact_columns(case, seed):
    zeta, c = geo.random_columns(case["nV"], case["nz"], seed=seed, stiff_frac=case["stiff"], stiffness=3000.0)
    nV, nz, DT, rho, T0, cc, sec = case["nV"], case["nz"], 5.0, 910.0, 273.16, 8.7e-4, geo.SEC_PER_YEAR
    H, mask, Ts = c["Hi_eff"], c["mask"], np.minimum(c["T_surf_annual"], T0)
    Ti, Q = c["Ti"], c["Q_base_grnd"]
    Cp = 2115.3 + 7.79293 * (Ti - T0)
    K = 3.101e8 * np.exp(-0.0057 * Ti)
    pmp = T0 - cc * H[:, None] * zeta[None, :]
    # derivative weights of three-point rows (second order on an irregular grid)
    l, u = np.zeros((2, nz)), np.zeros((2, nz))
    for k in range(1, nz - 1):
        h0, h1 = zeta[k - 1] - zeta[k], zeta[k + 1] - zeta[k]
        M = np.linalg.inv(np.array([[h0, h0 * h0 / 2], [h1, h1 * h1 / 2]]))
        l[:, k], u[:, k] = M[:, 0], M[:, 1]
    dg = -(l + u)
    c1 = c["dzeta_dt"] + c["u_3D"] * c["dzeta_dx"] + c["v_3D"] * c["dzeta_dy"] + c["w_3D"] * c["dzeta_dz"]
    c2 = -K / (rho * Cp) * c["dzeta_dz"] ** 2
    lo, di, up = (c1 * w[0] + c2 * w[1] for w in (l, dg, u))
    src = -c["u_times_dTdxp_upwind"] - c["v_times_dTdyp_upwind"] + c["internal_heating"] / (rho * Cp)
    grounded = (mask == pkg.abi.COL_GROUNDED) | (mask == pkg.abi.COL_GL_GR)

    def step(T, at, dt):
        lo_, di_, up_, B = lo[at], di[at], up[at], pmp[at, -1]
        flux = T[:, -2] - (zeta[-1] - zeta[-2]) * Q[at] / (c["dzeta_dz"][at, -1] * K[at, -1])
        base = np.where(grounded[at], np.minimum(B, flux), B)
        b, d = np.ones((len(at), nz)), np.empty((len(at), nz))
        d[:, 0] = Ts[at]
        up0 = np.zeros(len(at))
        for k in range(1, nz - 1):
            w = lo_[:, k] / b[:, k - 1]
            b[:, k] = 1.0 / dt + di_[:, k] - w * (up0 if k == 1 else up_[:, k - 1])
            d[:, k] = T[:, k] / dt + src[at, k] - w * d[:, k - 1]
        x = np.empty_like(T)
        x[:, -1] = base
        for k in range(nz - 2, -1, -1):
            x[:, k] = (d[:, k] - (up_[:, k] if k else 0.0) * x[:, k + 1]) / b[:, k]
        return np.minimum(x, pmp[at])

    bad = lambda x: (np.isnan(x) | (x < 180.0) | (x > T0)).any(1)  # noqa: E731
    out = np.repeat(c["T_surf_annual"][:, None], nz, 1)
    ice = np.nonzero(H >= 10.0)[0]
    with np.errstate(all="ignore"):
        out[ice] = step(Ti[ice], ice, DT)
        left = ice[bad(out[ice])]
        for lev in range(1, 10):
            if not len(left):
                break
            T = out[left]
            for _ in range(2 ** lev):
                T = step(T, left, DT * 0.5 ** lev)
            out[left] = T
            left = left[bad(T)]
    KR = 9.828 * sec * math.exp(-0.0057 * T0)
    for v in left:
        if grounded[v] and c["SMB"][v] > 0:
            L = math.sqrt(2.0 * KR / (rho * 2127.5) * H[v] / c["SMB"][v])
            e = np.array([math.erf((1.0 - z) * H[v] / L) - math.erf(H[v] / L) for z in zeta])
            t = Ts[v] - math.sqrt(math.pi) / 2.0 * L * c["geothermal_heat_flux"][v] / KR * e
        else:
            t = Ts[v] + ((T0 - cc * H[v]) - Ts[v]) * zeta
        out[v] = np.minimum(t, pmp[v])
    return out, int(len(left))


def _exact_network(case, seed):
    nbr = _graph(case["nTri"])
    flat, x, target, w = _network(len(nbr), nbr, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    flat = t(flat).double().requires_grad_(case["train"])
    P, at = {}, 0
    for name, shape in _LAYOUT:
        P[name] = flat[at:at + math.prod(shape)].view(shape)
        at += math.prod(shape)
    nb = t(nbr).long()
    there = (nb >= 0).double()
    h = torch.relu(t(x).double() @ P["We"].T + P["be"])
    for k in range(4):
        a = sum(h[nb[:, q].clamp(min=0)] * there[:, q:q + 1] for q in range(3)) / there.sum(1, keepdim=True).clamp(min=1.0)
        z = torch.relu(torch.cat([h, a], 1) @ P["W1%d" % k].T + P["b1%d" % k])
        h = h + z @ P["W2%d" % k].T + P["b2%d" % k]
    y = h @ P["Wd"].T + P["bd"]
    if not case["train"]:
        return y.cpu().numpy()
    loss = (t(w).double()[:, None] * (y - t(target).double()) ** 2).sum()
    loss.backward()
    return float(loss.detach()), flat.grad.cpu().numpy()
