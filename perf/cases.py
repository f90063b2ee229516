"""The work this framework is used for, as cases that can be timed.

A case names one of the kinds of call a user's program makes:

  rhs       one residual evaluation through the module procedure compute_rhs_ns, host
            buffers in and out: what a host code that keeps its own time loop calls per
            stage
  euler     a whole explicit solve: a device-resident state on a mesh the program keeps,
            n iterations of the time loop, the final state read back
  tubes     shock tubes of uneven length admitted to a batch engine the program keeps,
            advanced together until each reached its end time, read back and removed
  lagrange  n Lagrangian steps from the initial mesh and state, final state and vertex
            positions read back
  sedovs    Sedov problems of uneven size served together by the Lagrangian batch engine
  implicit  one backward-Euler Navier-Stokes step of a running state (assembly, GMRES,
            update), state read back
  gmres     one linear solve with a block matrix the program keeps on the device, host
            right-hand side in, solution out

Sizes and options come from the configurations, tests and benchmark of this repository.
"""
import math

import numpy as np

from subfv_b200 import meshgen, shocktube
from subfv_b200.bcsr import BcsrMatrix, DeviceBcsr
from subfv_b200.lagrange import LagBatch, LagrangeState, init_sol_sedov
from subfv_b200.mesh import Mesh
from subfv_b200.ns import NsBatch, NsConfig, NsState, compute_rhs_ns, init_fourier_flow, init_gresho
from subfv_b200.ns_init import init_sedov

# scheme ids of NsConfig
MULTI_POINT, TWO_WAVE = 1, 4
# the chunk of steps a program advances a batch by between looks at its problems
CHUNK = 8


def listed():
    return [
        # the smallest call: one residual of a small quadrilateral mesh, from a host code's own loop
        dict(name="rhs_quads_24x20", kind="rhs", mesh="quads", nx=24, ny=20, order=2, scheme=MULTI_POINT, precision=0),
        # the Gresho vortex at its configured size: second order, multi-point, 200 two-stage iterations
        dict(name="euler_gresho_quads_64", kind="euler", mesh="quads", flow="gresho", nx=64, ny=64, order=2,
             scheme=MULTI_POINT, precision=0, steps=200, viscous=""),
        # an ordinary second-order run on a triangle mesh that fills the GPU, ragged sides
        dict(name="euler_gresho_tris_39k", kind="euler", mesh="tris", flow="gresho", nx=149, ny=131, order=2,
             scheme=MULTI_POINT, precision=0, steps=24, viscous=""),
        # the explicit Sedov case at the reference's resolution: first order, two-wave flux, 29,282 triangles
        dict(name="euler_sedov_tris_121", kind="euler", mesh="tris", flow="sedov", nx=121, ny=121, order=1,
             scheme=TWO_WAVE, precision=0, steps=160, viscous=""),
        # three-dimensional explicit Navier-Stokes with a temperature-dependent viscosity, periodic box
        dict(name="euler_viscous_box_20", kind="euler", mesh="box", flow="fourier", nx=20, ny=20, order=2,
             scheme=MULTI_POINT, precision=0, steps=8, viscous="sutherland"),
        # a batch of shock tubes in plain FP64 and one with FP32 wave-speed bounds
        dict(name="tubes_64_fp64", kind="tubes", count=64, n_max=2000, order=1, scheme=MULTI_POINT, precision=0,
             t_scale=0.02),
        dict(name="tubes_96_mixed", kind="tubes", count=96, n_max=2000, order=1, scheme=MULTI_POINT, precision=1,
             t_scale=0.02),
        # the Lagrangian Sedov blast at its configured size (524,288 triangles), and a small one
        dict(name="lagrange_sedov_tris_512", kind="lagrange", mesh="tris", nx=512, ny=512, precision=0, steps=96),
        dict(name="lagrange_sedov_tris_40", kind="lagrange", mesh="tris", nx=41, ny=37, precision=0, steps=256),
        # served Lagrangian requests of uneven size, solved together
        dict(name="sedovs_24", kind="sedovs", count=24, cells_min=4096, cells_max=20000, precision=0, steps=64),
        # a backward-Euler Navier-Stokes step of a periodic box, block-Jacobi GMRES(30)
        dict(name="implicit_box_40", kind="implicit", nx=40, viscous="constant", refine=False, precond=1),
        # the linear solver alone on a 7-point matrix of 5x5 blocks
        dict(name="gmres_7pt_40", kind="gmres", nx=40, ny=40, nz=37, stencil=7, bs=5, precond=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "euler", "euler", "euler", "tubes", "lagrange", "lagrange", "sedovs", "implicit", "gmres"])
    if kind == "rhs":
        mesh = rng.choice(["quads", "tris", "box"])
        n = _log_int(rng, 6, 22) if mesh == "box" else _log_int(rng, 12, 150)
        return dict(kind=kind, mesh=mesh, nx=n, ny=max(4, n - rng.randrange(0, 7)), order=rng.choice([1, 2]),
                    scheme=rng.choice([MULTI_POINT, TWO_WAVE]), precision=rng.choice([0, 0, 1, 2]))
    if kind == "euler":
        mesh = rng.choice(["quads", "tris", "box"])
        n = _log_int(rng, 8, 30) if mesh == "box" else _log_int(rng, 20, 170)
        viscous = rng.choice(["", "", "constant", "sutherland"]) if n <= 20 and mesh == "box" else ""
        flow = "fourier" if mesh == "box" else rng.choice(["gresho", "sedov"]) if mesh == "tris" else "gresho"
        return dict(kind=kind, mesh=mesh, flow=flow, nx=n, ny=n if mesh == "box" else n + rng.randrange(0, 9),
                    order=rng.choice([1, 2]), scheme=rng.choice([MULTI_POINT, MULTI_POINT, TWO_WAVE]),
                    precision=0 if viscous else rng.choice([0, 0, 1, 2]), steps=8 if viscous else rng.randrange(20, 61),
                    viscous=viscous)
    if kind == "tubes":
        order = rng.choice([1, 1, 2])
        return dict(kind=kind, count=_log_int(rng, 4, 90 if order == 1 else 20), n_max=_log_int(rng, 400, 2000),
                    order=order, scheme=MULTI_POINT, precision=rng.choice([0, 1, 2]), t_scale=rng.uniform(0.008, 0.02))
    if kind == "lagrange":
        n = _log_int(rng, 16, 400)
        return dict(kind=kind, mesh=rng.choice(["tris", "tris", "quads"]), nx=n, ny=n + rng.randrange(0, 9),
                    precision=rng.choice([0, 0, 1]), steps=rng.randrange(30, 100))
    if kind == "sedovs":
        return dict(kind=kind, count=_log_int(rng, 2, 24), cells_min=1024, cells_max=_log_int(rng, 2048, 20000),
                    precision=rng.choice([0, 1]), steps=rng.randrange(20, 65))
    if kind == "implicit":
        return dict(kind=kind, nx=_log_int(rng, 8, 36), viscous=rng.choice(["", "constant"]),
                    refine=rng.random() < 0.3, precond=rng.choice([1, 1, 2]))
    n = _log_int(rng, 8, 40)
    stencil = 7 if n > 24 else rng.choice([7, 27])
    return dict(kind="gmres", nx=n, ny=max(4, n - rng.randrange(0, 4)), nz=max(4, n - rng.randrange(0, 4)),
                stencil=stencil, bs=rng.choice([4, 5, 5]), precond=rng.choice([0, 1, 1]))


# ---- inputs

def _raw(mesh, nx, ny, seed, lo=-0.5, hi=0.5, jitter=0.1):
    if mesh == "quads":
        return meshgen.hex_slab(nx, ny, lo, hi, lo, hi, -0.5, 0.5, jitter=jitter, seed=seed)
    if mesh == "tris":
        return meshgen.prism_slab(nx, ny, lo, hi, lo, hi, -0.5, 0.5, jitter=0.5 * jitter, seed=seed)
    return meshgen.hex_box(nx, jitter=0.5 * jitter, seed=seed, periodic=True)


def _perturbed(sol, seed, amp=1e-3):
    """Density and energy of every cell off by up to `amp` relative, from the seed."""
    f = 1.0 + amp * np.random.default_rng(seed).uniform(-1.0, 1.0, (sol.shape[0], 1))
    return np.ascontiguousarray(sol * f)


def _config(case, tmax=1e30):
    flat = case.get("mesh", "quads") != "box"
    kw = dict(scheme=case["scheme"], second_order=case["order"] == 2, method=4 if case["order"] == 2 else 0, bc_style=2,
              boundary_2d=flat, cfl=0.4, precision=case["precision"], tmax=tmax)
    if case.get("viscous") == "constant":
        kw.update(activate_diffusion=True, mu_p=1e-3, prandtl=0.72)
    elif case.get("viscous") == "sutherland":  # reference temperature and viscosity scaled to the flow's
        kw.update(activate_diffusion=True, use_sutherland=True, mu0=1e-3, T0=0.01, prandtl=0.72)
    return NsConfig(**kw)


def _flow(case, mesh, seed):
    if case["mesh"] == "box":
        return init_fourier_flow(mesh, seed=seed)
    if case.get("flow") == "sedov":
        return _perturbed(init_sedov(mesh.geometry("elem_coord"), mesh.geometry("elem_volume")), seed)
    return _perturbed(init_gresho(mesh, 0.1), seed)


def _sedov(mesh):
    t = mesh.topo
    mask = meshgen.sedov_origin_mask(t.array("elem_vert_off"), t.array("elem_vert"), t.coords())
    sol = init_sol_sedov(mesh, e_total=0.244816, mask=mask)
    return sol, mesh.geometry("elem_volume") / sol[:, 0]


def _sedov_sizes(case):
    """Squares per side of the requests: cell counts spread over the logarithm of the range."""
    lo, hi, n = math.log(case["cells_min"]), math.log(case["cells_max"]), case["count"]
    return [max(4, int(round(math.sqrt(math.exp(lo + (hi - lo) * (i + 0.5) / n) / 2)))) for i in range(n)]


def _tubes(case, seed):
    """Seeded tubes; their lengths are the case's own, so that every seed has the same work."""
    sizes = np.random.default_rng(case["count"] * 100003 + case["n_max"]).integers(200, case["n_max"] + 1, case["count"])
    tubes = shocktube.sample(case["count"], seed=seed, n_max=case["n_max"])
    return [shocktube.ShockTube(int(n), t.left, t.right, t.t_end) for n, t in zip(sizes, tubes)]


def _matrix(case, seed):
    """Blocks of the 7- or 27-point neighbours of a grid, ascending columns, with a block
    diagonal that dominates as V/dt does in an implicit step."""
    nx, ny, nz, bs = case["nx"], case["ny"], case["nz"], case["bs"]
    rng = np.random.default_rng(seed)
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    m = nx * ny * nz
    cols, valid = [], []
    for dk in (-1, 0, 1):
        for dj in (-1, 0, 1):
            for di in (-1, 0, 1):
                if case["stencil"] == 7 and abs(di) + abs(dj) + abs(dk) > 1:
                    continue
                a, b, c = i + di, j + dj, k + dk
                valid.append((a >= 0) & (a < nx) & (b >= 0) & (b < ny) & (c >= 0) & (c < nz))
                cols.append((c * ny + b) * nx + a)
    valid, cols = np.stack(valid, 1), np.stack(cols, 1)
    row = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    col = cols[valid].astype(np.int32)
    v = rng.uniform(-1.0, 1.0, (col.size, bs, bs))
    v *= 1.0 / case["stencil"]
    v[col == np.repeat(np.arange(m), np.diff(row))] += 1.5 * np.eye(bs)
    return BcsrMatrix(m, bs, row + 1, col + 1, v), rng.standard_normal(m * bs)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rhs", "euler"):
        mesh = Mesh.from_raw(_raw(case["mesh"], case["nx"], case["ny"], seed))
        return dict(kind=kind, mesh=mesh, cfg=_config(case), sol=_flow(case, mesh, seed), steps=case.get("steps", 0))
    if kind == "tubes":
        tubes = _tubes(case, seed)
        meshes = [Mesh.from_raw(shocktube.raw_mesh(t)) for t in tubes]
        # room for the problems that leave while the next ones are admitted
        batch = NsBatch(_config(case), capacity=2 * case["count"], budget_bytes=int(20e9))
        return dict(kind=kind, batch=batch, problems=[
            (m, shocktube.initial_state(m, t), t.t_end * case["t_scale"]) for m, t in zip(meshes, tubes)])
    if kind == "lagrange":
        mesh = Mesh.from_raw(_raw(case["mesh"], case["nx"], case["ny"], seed, 0.0, 1.2))
        sol, mass = _sedov(mesh)
        state = LagrangeState(mesh, sol, mass, cfl=0.5, t_max=1e30, precision=case["precision"])
        return dict(kind=kind, mesh=mesh, state=state, coords=mesh.coords(), sol=sol, steps=case["steps"])
    if kind == "sedovs":
        batch = LagBatch(capacity=2 * case["count"], budget_bytes=int(20e9), precision=case["precision"])
        problems = []
        for i, n in enumerate(_sedov_sizes(case)):
            mesh = Mesh.from_raw(_raw("tris", n, n, seed * 64 + i, 0.0, 1.2))
            problems.append((mesh, mesh.coords()) + _sedov(mesh))
        return dict(kind=kind, batch=batch, problems=problems, steps=case["steps"])
    if kind == "implicit":
        mesh = Mesh.from_raw(_raw("box", case["nx"], case["nx"], seed))
        cfg = _config(dict(case, mesh="box", scheme=TWO_WAVE, order=1, precision=0))
        state = NsState(mesh, cfg, init_fourier_flow(mesh, seed=seed))
        return dict(kind=kind, state=state, refine=case["refine"], precond=case["precond"])
    A, b = _matrix(case, seed)
    return dict(kind=kind, A=DeviceBcsr(A), b=b, tol=1e-10 * float(np.linalg.norm(b)), precond=bool(case["precond"]))


# ---- one pass

def run(state):
    kind = state["kind"]
    if kind == "rhs":
        status, rhs, sum_lambda, vp, grad = compute_rhs_ns(state["mesh"], state["cfg"], state["sol"])
        return dict(status=status, rhs=rhs, sum_lambda=sum_lambda, vp=vp, grad=grad)
    if kind == "euler":
        s = NsState(state["mesh"], state["cfg"], state["sol"])
        status, steps, t = s.advance(state["steps"])
        out = dict(status=status, steps=steps, t=t, sol=s.sol())
        s.close()
        return out
    if kind == "tubes":
        batch = state["batch"]
        slots = [batch.add(m, sol, t_end) for m, sol, t_end in state["problems"]]
        info = []
        while not info or not all(done or status for _, _, done, status in info):
            batch.advance(CHUNK)
            batch.sync()
            info = [batch.info(k) for k in slots]
        sols = [batch.sol(k, m.n_elems) for k, (m, _, _) in zip(slots, state["problems"])]
        for k in slots:
            batch.remove(k)
        return dict(sol=np.concatenate(sols), t=np.array([i[0] for i in info]), steps=np.array([i[1] for i in info]),
                    status=np.array([i[3] for i in info]))
    if kind == "lagrange":
        mesh, s = state["mesh"], state["state"]
        mesh.set_coords(state["coords"])
        mesh.compute_geometry_mesh()
        s.set_sol(state["sol"])
        status, _, _ = s.advance(state["steps"])
        return dict(status=status, sol=s.sol(), coords=mesh.coords(), dt=s.last_dt())
    if kind == "sedovs":
        batch, slots = state["batch"], []
        for mesh, coords, sol, mass in state["problems"]:
            mesh.set_coords(coords)
            mesh.compute_geometry_mesh()
            slots.append(batch.add(mesh, sol, 1e30, cfl=0.5, mass=mass))
        batch.advance(state["steps"])
        batch.sync()
        info = [batch.info(k) for k in slots]
        sols = [batch.sol(k, p[0].n_elems) for k, p in zip(slots, state["problems"])]
        for k in slots:
            batch.remove(k)
        return dict(sol=np.concatenate(sols), t=np.array([i[0] for i in info]), steps=np.array([i[1] for i in info]),
                    status=np.array([i[3] for i in info]))
    if kind == "implicit":
        s = state["state"]
        status, stats = s.implicit_step(cfl_implicit=10.0, refine_fp32=state["refine"], precond=state["precond"])
        return dict(status=status, dt=stats["dt"], sol=s.sol())
    x, conv, _, rho = state["A"].gmres(state["b"], state["tol"], m=30, precond=state["precond"])
    return dict(x=x, converged=conv)


# ---- what a pass cannot do without

# operations of one subface in one residual: the states' primitives and wave speeds, the
# nodal solver's four iterations (one for two-wave), the flux pair and its sums
_FLOPS_SUBFACE = {MULTI_POINT: 500.0, TWO_WAVE: 150.0}
# cells, vertices and subfaces of a mesh of n cells: subcells per cell, subfaces per cell, vertices per cell
_SHAPE = {"quads": (8.0, 16.0, 2.0), "tris": (6.0, 12.0, 1.0), "box": (8.0, 12.0, 1.0)}


def _cells(case):
    n = case["nx"] * case["ny"]
    return {"quads": n, "tris": 2 * n, "box": case["nx"] ** 3}[case["mesh"]]


def _euler_work(case, cells, mesh, evaluations):
    """Per residual evaluation: the state in and out, the vertex positions, the cells'
    vertex and face lists; operations of the fluxes, once more per order."""
    vc, sf, nv = _SHAPE[mesh]
    per = 80.0 + 24.0 * nv + 4.0 * (vc + 6.0)
    return {"bytes": evaluations * cells * per,
            "flops": evaluations * cells * sf * _FLOPS_SUBFACE[case["scheme"]] * case["order"]}


def _lagrange_work(mesh, cells, steps):
    """Per step: the state and the vertex positions in and out, the cells' lists; the face
    and subcell geometry, nodal system and fluxes of every subface."""
    vc, sf, nv = _SHAPE[mesh]
    return {"bytes": steps * cells * (80.0 + 48.0 * nv + 4.0 * (vc + 6.0)), "flops": steps * cells * sf * 250.0}


def _gmres_work(nnz_blocks, rows, bs, krylov, cycles):
    """Per restart cycle: krylov products with the matrix, and each basis vector read once
    for every later column's projections."""
    n = rows * bs
    return {"bytes": cycles * (krylov * (nnz_blocks * (8.0 * bs * bs + 4.0) + 8.0 * rows * bs * bs)
                               + 8.0 * n * krylov * (krylov + 1) / 2),
            "flops": cycles * (krylov * 2.0 * nnz_blocks * bs * bs + 4.0 * n * krylov * (krylov + 1) / 2)}


def work(case):
    kind = case["kind"]
    if kind == "rhs":
        cells = _cells(case)
        w = _euler_work(case, cells, case["mesh"], 1)
        w["bytes"] += 8.0 * cells * (6 + 15 + 3)  # the gradients, residuals and velocities go back to the host
        return w
    if kind == "euler":
        w = _euler_work(case, _cells(case), case["mesh"], case["steps"] * case["order"])
        if case["viscous"]:  # the nodes' 36 x 36 momentum and 12 x 12 heat systems, inverted and applied
            w["flops"] += case["steps"] * case["order"] * _cells(case) * 4.0 * 36 ** 3
        return w
    if kind == "tubes":
        sizes = [t.n for t in _tubes(case, 1)]
        # the step count of a tube grows with its length: t_scale * 0.25 / cfl * n
        return _euler_work(case, sum(4.0 * n * case["order"] * max(1.0, case["t_scale"] * 0.25 / 0.4 * n)
                                     for n in sizes), "quads", 1)
    if kind == "lagrange":
        return _lagrange_work(case["mesh"], _cells(case), case["steps"])
    if kind == "sedovs":
        return _lagrange_work("tris", sum(2 * n * n for n in _sedov_sizes(case)), case["steps"])
    if kind == "implicit":
        cells = case["nx"] ** 3
        w = _gmres_work(7 * cells, cells, 5, 30, 1)
        w["bytes"] += 8.0 * (175.0 + 10.0) * cells  # the Jacobian written once, the state in and out
        w["flops"] += cells * 12.0 * 600.0
        return w
    rows = case["nx"] * case["ny"] * case["nz"]
    return _gmres_work(case["stencil"] * rows, rows, case["bs"], 30, 1)


# ---- reference values in 64 bits

def _gmres_numpy(A, b, tol):
    """x with |b - A x| <= tol by flexible restarted GMRES with a block-diagonal
    preconditioner, all in numpy."""
    m, bs = A.m, A.blc_size
    row, col = np.asarray(A.row) - 1, np.asarray(A.col) - 1
    rows = np.repeat(np.arange(m), np.diff(row))
    blocks = A.v.transpose(0, 2, 1)  # [j, r, c]
    dinv = np.linalg.inv(blocks[rows == col])

    def mul(x):
        y = np.einsum("jrc,jc->jr", blocks, x.reshape(m, bs)[col])
        return np.add.reduceat(y, row[:-1], axis=0).ravel()

    def pre(x):
        return np.einsum("irc,ic->ir", dinv, x.reshape(m, bs)).ravel()

    x = np.zeros(m * bs)
    for _ in range(20):
        r = b - mul(x)
        beta = np.linalg.norm(r)
        if beta <= tol:
            break
        V, Z, H = [r / beta], [], np.zeros((21, 20))
        for j in range(20):
            Z.append(pre(V[j]))
            w = mul(Z[j])
            for i in range(j + 1):
                H[i, j] = w @ V[i]
                w -= H[i, j] * V[i]
            H[j + 1, j] = np.linalg.norm(w)
            V.append(w / H[j + 1, j])
        y = np.linalg.lstsq(H, beta * np.eye(21)[:, 0], rcond=None)[0]
        x = x + sum(c * z for c, z in zip(y, Z))
    return x


def exact(case, seed):
    # The solvers of the other kinds are their own definition: a scheme on an unstructured
    # mesh in this framework's numbering has no value in 64 bits apart from this code.
    if case["kind"] != "gmres" or case["nx"] * case["ny"] * case["nz"] * case["stencil"] > 5e5:
        return None
    A, b = _matrix(case, seed)
    return dict(x=_gmres_numpy(A, b, 1e-14 * float(np.linalg.norm(b))), converged=None)
