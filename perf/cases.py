"""Workloads of the engine as a user's program runs them, for measuring speed and accuracy.

Every case goes through the public entry points: the solver classes and problem
builders (load steps), BatchedBlocks with DisplacementMisfit (a load ramp and
the gradient of its misfit) and return_mapping (batches of material points).

A pass of a load-step case puts the solver back to the start of a ramp (which
is what an inverse analysis does before each gradient, and a time stepper
before it repeats a rejected step) and runs `steps` load steps from there; the
updated particle state comes back, and the loss and gradient where there is an
adjoint.
"""
import math

import numpy as np
import torch

from geowarp_b200 import problems
from geowarp_b200.adjoint import DisplacementMisfit
from geowarp_b200.batch import BatchedBlocks
from geowarp_b200.materials.plasticity import return_mapping
from geowarp_b200.solvers.quasi_static_coupled_solver_2d import quasi_static_coupled_solver_2d

NU = 0.3

# NorSand: the loose Brasted sand of the triaxial material test
NORSAND = dict(kappa=0.0015, tilde_lambda=0.02, M=1.27, N=0.4, beta=1.0, vc0=1.8911, p0=-390.0, v0=1.75, h=70.0,
               shear_modulus=4.5e4)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the bar under self-weight, the reference's own small problem: hundreds
        # of particles, where the step is launches and host reads
        dict(name="bar_4x40_fp64", family="bar", nx=4, ny=40, material="Neo-Hookean", precision="fp64", steps=1),
        # a wider plastic bar in mixed precision: J2 return map, and the second
        # step starts from the first one's increment
        dict(name="bar_13x71_j2_mixed", family="bar", nx=13, ny=71, material="J2", precision="mixed", steps=2),
        # inverse analysis of one block, FP64: ramp and gradient
        dict(name="block_47x33_fp64_grad", family="blocks", n=1, nx=47, ny=33, precision="fp64", steps=2, grad=True),
        # a plain forward run of a few blocks in FP64 (the drop-in precision)
        dict(name="blocks_8_fp64", family="blocks", n=8, nx=96, ny=56, precision="fp64", steps=1, grad=False),
        # forward ramp of a batch in mixed precision (generating targets)
        dict(name="blocks_16_mixed", family="blocks", n=16, nx=128, ny=64, precision="mixed", steps=2, grad=False),
        # the benchmark's batched inverse analysis: 64 blocks, ramp and gradient
        dict(name="blocks_64_mixed_grad", family="blocks", n=64, nx=128, ny=64, precision="mixed", steps=2, grad=True),
        # strip footing on Drucker-Prager soil at the benchmark's size
        dict(name="footing_256x128_fp64", family="footing", nx=256, ny=128, precision="fp64"),
        # a smaller footing with an odd cell count in mixed precision
        dict(name="footing_97x51_mixed", family="footing", nx=97, ny=51, precision="mixed"),
        # one-dimensional consolidation (u-p) at the benchmark's size
        dict(name="column_200_fp64", family="column", nx=1, ny=200, material="Linear elasticity", precision="fp64",
             law="constant", projection="consistent", steps=2),
        # a wide consolidating layer (u-p), mixed precision, with the
        # deformation-dependent mobility and the lumped projection
        dict(name="layer_63x40_mixed", family="column", nx=63, ny=40, material="Neo-Hookean", precision="mixed",
             law="Uzuoka-Borja", projection="lumped", steps=1),
        # three-dimensional indentation (u-p), one load step
        dict(name="indentation_5_fp64", family="indentation", nx=5, ny=5, nz=5, precision="fp64"),
        # material points of a Drucker-Prager soil with their tangents
        dict(name="points_dp_1m", family="points", material="Drucker-Prager", n=1000003, tangent=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["bar", "blocks", "blocks", "footing", "column", "indentation", "points"])
    precision = rng.choice(["fp64", "mixed"])
    if family == "bar":
        return dict(family=family, nx=_log_int(rng, 2, 24), ny=_log_int(rng, 10, 120),
                    material=rng.choice(["Neo-Hookean", "Hencky elasticity", "J2", "Linear elasticity"]),
                    precision=precision, steps=rng.choice([1, 2]))
    if family == "blocks":
        return dict(family=family, n=_log_int(rng, 1, 24), nx=rng.randint(16, 128), ny=rng.randint(16, 64),
                    precision=precision, steps=rng.choice([1, 2]), grad=rng.random() < 0.5)
    if family == "footing":
        ny = rng.randint(32, 128)
        return dict(family=family, nx=rng.randint(max(48, ny), 256), ny=ny, precision=precision)
    if family == "column":
        nx = rng.choice([1, rng.randint(2, 64)])
        ny = _log_int(rng, 20, 300) if nx == 1 else rng.randint(12, 48)
        return dict(family=family, nx=nx, ny=ny, material=rng.choice(["Linear elasticity", "Neo-Hookean"]),
                    precision=precision, law=rng.choice(["constant", "Uzuoka-Borja"]),
                    projection=rng.choice(["consistent", "lumped"]), steps=rng.choice([1, 2]))
    if family == "indentation":
        return dict(family=family, nx=rng.randint(3, 6), ny=rng.randint(3, 6), nz=rng.randint(3, 6), precision="fp64")
    return dict(family=family, material=rng.choice(["J2", "Drucker-Prager", "NorSand"]), n=_log_int(rng, 1, 1000000),
                tangent=rng.random() < 0.5)


# ---------------------------------------------------------------- inputs
def _log_field(x, seed, mean, std=0.3, corr=0.5):
    """log E at particle positions x [N, 2]: a smooth random field (a sum of
    random cosines with a Gaussian spectrum of correlation length corr)."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    k = torch.randn((48, 2), generator=g, dtype=torch.float64) * (math.sqrt(2.0) / corr)
    ph = torch.rand(48, generator=g, dtype=torch.float64) * (2.0 * math.pi)
    k, ph = k.to(x.device), ph.to(x.device)
    out = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
    for q in range(48):
        out += torch.cos(x[:, 0] * k[q, 0] + x[:, 1] * k[q, 1] + ph[q])
    return mean + std * math.sqrt(2.0 / 48) * out


def _sizes(case):
    """Cell counts of a batch's blocks: the first is the largest, the others
    spread down to a quarter of its width and half its height."""
    r = np.random.default_rng(1000 * case["nx"] + 10 * case["ny"] + case["n"])
    nx = r.integers(max(2, case["nx"] // 4), case["nx"] + 1, size=case["n"])
    ny = r.integers(max(2, case["ny"] // 2), case["ny"] + 1, size=case["n"])
    nx[0], ny[0] = case["nx"], case["ny"]
    return [(int(a), int(b)) for a, b in zip(nx, ny)]


BAR_RAMP = 4      # load steps of the bar's ramp
BLOCK_RAMP = 100  # load steps of the blocks' ramp
KAPPA = 1500.0    # yield stress of the J2 bar, reached in its lower half


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    fam = case["family"]
    dev = torch.device("cuda", torch.cuda.current_device())
    st = dict(case=case)
    if fam == "points":
        return _prepare_points(case, seed, dev, st)
    if fam == "bar":
        mat = case["material"]
        s = problems.bar_compaction_2d(precision=case["precision"], width_cells=case["nx"], height_cells=case["ny"],
                                       dx=0.25, material="Hencky elasticity" if mat == "J2" else mat,
                                       tol=1e-6)
        if mat == "J2":  # the builder has no yield stress: the same set-up with the material replaced
            s = _j2_bar(s, case)
        st["logE"] = _log_field(s.x_particles, seed, math.log(1e6), corr=2.0)
        s.engine.E = torch.exp(st["logE"])
    elif fam == "blocks":
        bb = BatchedBlocks(_sizes(case), precision=case["precision"])
        s, st["blocks"] = bb.solver, bb
        st["logE"] = _log_field(s.x_particles, seed, math.log(1e7))
        s.engine.E = torch.exp(st["logE"])
        if case["grad"]:
            st["logE"].requires_grad_(True)
            t = _log_field(s.x_particles, seed + 7919, 0.0)
            st["target"] = torch.stack([1e-4 * t, -5e-4 * torch.exp(t)], 1)
    elif fam == "footing":
        s = problems.strip_footing_2d(precision=case["precision"], n_cells_x=case["nx"], n_cells_y=case["ny"],
                                      E=2e7 * math.exp(0.2 * rng.standard_normal()),
                                      cohesion=1e4 * math.exp(0.1 * rng.standard_normal()))
    elif fam == "column":
        s, st["dts"], st["n_steps"] = _column(case, rng)
    else:
        block = (case["nx"], case["ny"], case["nz"])
        s = problems.indentation_3d(precision=case["precision"], precond="block", block_cells=block,
                                    grid_cells=tuple(n + 2 for n in block), dx=0.25,
                                    E=1e3 * math.exp(0.2 * rng.standard_normal()), material="Neo-Hookean",
                                    permeability=1e-11, indenter=0.5, depth=0.5, n_steps=25, penalty=1000.0)
    st["solver"] = s
    arrays = [s.x_particles, s.GIMP_lp, s.deformation_gradient_total_old, s.deformation_gradient_total_new,
              s.left_Cauchy_Green_old, s.left_Cauchy_Green_new, s.particle_Cauchy_stress_array]
    if fam in ("column", "indentation"):
        arrays.append(s.particle_pressure_array)
    st["start"] = [(a, a.clone()) for a in arrays]
    return st


def _j2_bar(s, case):
    from geowarp_b200.solvers.quasi_static_solver_2d import quasi_static_solver_2d
    dx, pad = 0.25, 2
    grid = dict(n_grid_x=s.n_grid_x, n_grid_y=s.n_grid_y, max_x=s.n_grid_x * dx, dx=dx, start_x=pad * dx,
                end_x=(pad + case["nx"]) * dx, start_y=pad * dx, end_y=(pad + case["ny"]) * dx,
                domain_min_x=pad * dx, domain_max_x=(pad + case["nx"]) * dx, domain_min_y=pad * dx,
                domain_max_y=(pad + case["ny"]) * dx)
    parts = dict(n_particles=s.n_particles, PPD=2, p_vol=s.p_vol, p_rho=s.p_rho)
    mat = dict(youngs_modulus=1e6, poisson_ratio=NU, material_name="J2", kappa=KAPPA)
    load = dict(gravity_mag=s.gravity_mag)
    t = quasi_static_solver_2d(grid, parts, dict(n_iter=20, tol=1e-6), mat, load, precision=case["precision"])
    t.dofStruct.boundary_flag_array.copy_(s.dofStruct.boundary_flag_array)
    return t


def _column(case, rng):
    """A consolidating layer nx cells wide (nx = 1: the column) under a surface
    load, drained at the top: the column builder's set-up, widened."""
    n_steps = 100
    E = 1e7 * math.exp(0.2 * rng.standard_normal())
    q = 1e4 * math.exp(0.2 * rng.standard_normal())
    grid, parts, it, mat, porous, load, dts, _, _ = problems.consolidation_column_dicts(
        n_cells=case["ny"], n_steps=n_steps, E=E, surface_load=q, material=case["material"], first_fourier=4.0)
    nx, dx = case["nx"], grid["dx"]
    grid.update(n_grid_x=nx + 5, max_x=(nx + 5) * dx, end_x=(nx + 1) * dx, domain_max_x=(nx + 1) * dx)
    parts["n_particles"] *= nx
    porous.update(mobility_law=case["law"], p2g_projection=case["projection"])

    def walls(tid, flags, n_grid_x, n_nodes):
        ix, iy = tid
        dof = ix + iy * (n_grid_x + 1)
        flags[dof[(ix <= 1) | (ix >= nx + 1)]] = True
        flags[dof[iy <= 0] + n_nodes] = True

    s = quasi_static_coupled_solver_2d(grid, parts, it, mat, porous, load, walls, precision=case["precision"],
                                       precond="mg")
    if case["precision"] == "fp64":
        s.engine.krylov_rtol = 1e-10  # as the column builder sets it
    top = s.x_particles[:, 1] > grid["end_y"] - dx / parts["PPD"]
    s.particle_pressure_boundary_flag_array[:] = top
    s.particle_traction_flag_array[:] = top
    return s, dts, n_steps


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    fam = case["family"]
    if fam == "points":
        e, tau, dtau, pi = return_mapping(state["material"], state["e_trial"], tangent=case["tangent"], **state["more"])
        return dict(e=e, tau=tau, dtau=dtau, pi=pi)
    s = state["solver"]
    for a, a0 in state["start"]:
        a.copy_(a0)
    if fam == "blocks" and case["grad"]:
        logE = state["logE"]
        logE.grad = None
        loss = DisplacementMisfit.apply(logE, s, state["target"], BLOCK_RAMP, case["steps"],
                                        lambda _: state["blocks"].reset_state())
        loss.backward()
        return dict(_solid(s), loss=loss.detach(), grad=logE.grad)
    if fam in ("bar", "blocks"):
        for k in range(case["steps"]):
            s.advance_one_step(k, BAR_RAMP if fam == "bar" else BLOCK_RAMP)
        return _solid(s)
    if fam == "footing":
        s.advance_one_step(0, 100)
        return dict(_solid(s), force=s.engine.force)
    if fam == "column":
        for k in range(case["steps"]):
            s.dt = float(state["dts"][k])
            s.advance_one_step(k, state["n_steps"])
        return dict(_solid(s), pressure=s.particle_pressure_array)
    s.advance_one_step(0, 25)
    return dict(_solid(s), pressure=s.particle_pressure_array, force=float(s.indentation_force[0]))


def _solid(s):
    return dict(x=s.x_particles, lp=s.GIMP_lp, F=s.deformation_gradient_total_old, b=s.left_Cauchy_Green_old,
                sigma=s.particle_Cauchy_stress_array)


def _particles(case):
    fam = case["family"]
    if fam == "points":
        return case["n"]
    if fam == "blocks":
        return 4 * sum(a * b for a, b in _sizes(case))
    if fam == "indentation":
        return 8 * case["nx"] * case["ny"] * case["nz"]
    return 4 * case["nx"] * case["ny"]


def work(case):
    """Bytes: the particle state in and out once per pass (and the gradient's
    inputs and outputs); operations: one residual and tangent evaluation per
    load step, about 1,500 per particle in 2D and 6,000 in 3D."""
    N = _particles(case)
    if case["family"] == "points":
        return dict(bytes=N * 8.0 * (3 + 6 + (9 if case["tangent"] else 0)), flops=N * 200.0)
    D = 3 if case["family"] == "indentation" else 2
    up = case["family"] in ("column", "indentation")
    steps = case.get("steps", 1)
    nbytes = N * 8.0 * ((2 * D + 18 + 1 + up) + (2 * D + 27 + up))
    flops = N * steps * (1500.0 if D == 2 else 6000.0)
    if case.get("grad"):
        nbytes += N * 8.0 * (1 + 2 + 1)  # log E and targets in, gradient out
        flops *= 2
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------- material points
def _prepare_points(case, seed, dev, st):
    g = torch.Generator(device=dev).manual_seed(seed)
    n, mat = case["n"], case["material"]
    z = torch.randn((n, 3), generator=g, dtype=torch.float64, device=dev)
    st["more"] = {}
    if mat == "NorSand":
        # the K0-consolidated state with small compressive / deviatoric increments
        p = dict(NORSAND)
        K = p["p0"] / (-p["kappa"])
        lam, mu = K - 2.0 / 3.0 * p["shear_modulus"], p["shear_modulus"]
        slope = (1.0 - 0.45) / ((1.0 + 2.0 * 0.45) / 3.0)
        txx = (3.0 - slope) / 3.0 * p["p0"]
        tau = np.array([txx, txx, (3.0 + 2.0 * slope) / 3.0 * p["p0"]])
        e0 = np.linalg.solve(lam * np.ones((3, 3)) + 2.0 * mu * np.eye(3), tau)
        r = torch.rand((n, 3), generator=g, dtype=torch.float64, device=dev)
        e = torch.as_tensor(e0, device=dev) + r * torch.tensor([4e-4, 4e-4, -3e-3], dtype=torch.float64, device=dev)
        pi0 = -715.0 * (1.0 - p["N"]) ** ((1.0 - p["N"]) / p["N"])
        pi = torch.full((n,), pi0, dtype=torch.float64, device=dev)
        st["material"] = dict(material_name="NorSand", initial_volumetric_strain=float(e0.sum()), **p)
        st["more"] = dict(eps_v_total=e.sum(1), pi_old=pi, pi_new=pi.clone())
    elif mat == "J2":
        e = 2e-3 * z
        st["material"] = dict(material_name="J2", youngs_modulus=1e6, poisson_ratio=NU, kappa=KAPPA)
    else:  # compressed soil with a shear that yields about half of the points
        e = 3e-3 * (z - z.mean(1, keepdim=True)) - 5e-4
        st["material"] = dict(material_name="Drucker-Prager", youngs_modulus=2e7, poisson_ratio=NU,
                              friction_angle=30.0, dilation_angle=5.0, cohesion=1e4, shape_factor=0.0)
    st["e_trial"] = e
    return st


def _exact_points(case, st):
    """Closed-form returns: J2, and the Drucker-Prager cone (shape factor 0)."""
    m, etr = st["material"], st["e_trial"]
    E, nu = m["youngs_modulus"], m["poisson_ratio"]
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    K = lam + 2.0 * mu / 3.0
    one = torch.ones(3, dtype=torch.float64, device=etr.device)
    tau_tr = lam * etr.sum(1, keepdim=True) + 2.0 * mu * etr
    P = tau_tr.mean(1, keepdim=True)
    S = tau_tr - P
    nrm = S.norm(dim=1, keepdim=True)
    nh = S / nrm.clamp_min(1e-300)
    I = torch.eye(3, dtype=torch.float64, device=etr.device)
    dev = I - 1.0 / 3.0
    nn = nh[:, :, None] * nh[:, None, :]
    Ce = lam * torch.ones_like(I) + 2.0 * mu * I
    if case["material"] == "J2":
        y = nrm - m["kappa"]
        dl = y / (2.0 * mu)
        e = etr - dl * nh
        d = Ce - 2.0 * mu * (nn + (dl * 2.0 * mu / nrm)[:, :, None] * (dev - nn))
        plastic = y > 0
    else:
        rad = 3.14159265358979 / 180.0
        s, c = math.sin(m["friction_angle"] * rad), math.cos(m["friction_angle"] * rad)
        sd = math.sin(m["dilation_angle"] * rad)
        A = 2.0 * math.sqrt(6.0) * m["cohesion"] * c / (3.0 - s)
        B = 2.0 * math.sqrt(6.0) * s / (3.0 - s)
        Bp = 2.0 * math.sqrt(6.0) * sd / (3.0 - sd)
        y = nrm - A + B * P
        den = 2.0 * mu + K * B * Bp
        dl = y / den
        e = etr - dl * (Bp / 3.0 * one + nh)
        ddl = (2.0 * mu * nh + B * K) / den  # d dl / d e_trial
        g = Bp / 3.0 * one + nh
        dn = 2.0 * mu / nrm[:, :, None] * (dev - nn)
        de = I - g[:, :, None] * ddl[:, None, :] - dl[:, :, None] * dn
        d = torch.matmul(Ce, de)
        plastic = (y >= 1e-10) & (P < 0)
        if bool((plastic & (nrm - 2.0 * mu * dl <= 0)).any()):
            return None  # beyond the cone's tip: no closed form
    e = torch.where(plastic, e, etr)
    tau = lam * e.sum(1, keepdim=True) + 2.0 * mu * e
    dt = torch.where(plastic[:, :, None], d, Ce.expand_as(d)) if case["tangent"] else None
    return dict(e=e, tau=tau, dtau=dt, pi=None)


# ---------------------------------------------------------------- 64-bit values of small solid ramps
MAX_EXACT_DOFS = 5000


def exact(case, seed):
    fam = case["family"]
    if fam == "points" and case["material"] != "NorSand":
        return _exact_points(case, prepare(case, seed))
    if fam not in ("bar", "blocks"):
        return None
    st = prepare(case, seed)
    s = st["solver"]
    bar = fam == "bar"
    d = _Dense(s.x_particles.clone(), s.GIMP_lp.clone(), s.deformation_gradient_total_old.clone(),
               s.left_Cauchy_Green_old.clone(), s.dofStruct.boundary_flag_array.clone(),
               h=s.dx, ncx=s.n_grid_x, ncy=s.n_grid_y, lp0=s.GIMP_lp_initial, V0=s.p_vol, rho=s.p_rho,
               g=s.gravity_mag, lo=(s.domain_min_x, s.domain_min_y), hi=(s.domain_max_x, s.domain_max_y),
               material=case["material"] if bar else "Hencky elasticity")
    if d.n_dofs > MAX_EXACT_DOFS:
        return None
    grad = bool(case.get("grad"))
    logE = st["logE"].detach().clone().requires_grad_(grad)
    E = torch.exp(logE)
    ramp = BAR_RAMP if bar else BLOCK_RAMP
    x0 = d.x
    q = (d.x, d.lp, d.F, d.b)
    for k in range(case["steps"]):
        q, sigma = d.step(q, E, (k + 1.0) / ramp)
    out = dict(x=q[0], lp=q[1], F=q[2], b=q[3], sigma=sigma)
    if grad:
        m = q[0] - x0 - st["target"]
        loss = 0.5 * (m * m).sum()
        loss.backward()
        out.update(loss=loss, grad=logE.grad)
    return {k: v.detach() for k, v in out.items()}


def _log_sym(b):
    """log of symmetric matrices near the identity: 2 artanh((b - I)(b + I)^-1)."""
    I = torch.eye(3, dtype=b.dtype, device=b.device)
    z = torch.linalg.solve(b + I, b - I)
    z2 = z @ z
    p, out = z, z
    for k in range(1, 12):
        p = p @ z2
        out = out + p / (2 * k + 1)
    return 2.0 * out


class _Dense:
    """Newton load steps of the 2D solid material-point formulation with a dense
    Jacobian, in plain torch; differentiable in E and the particle state (one
    further Newton update with the Jacobian held fixed carries the derivative
    of the implicit solution)."""

    def __init__(self, x, lp, F, b, fixed, h, ncx, ncy, lp0, V0, rho, g, lo, hi, material):
        self.x, self.lp, self.F, self.b = x, lp, F, b
        self.h, self.ncx, self.ncy, self.lp0, self.V0, self.rho, self.g = h, ncx, ncy, lp0, V0, rho, g
        self.lo, self.hi, self.material = lo, hi, material
        self.fixed = fixed
        self.nn = (ncx + 1) * (ncy + 1)
        W, _, nodes = self.shape(x, lp)
        active = torch.zeros(self.nn, dtype=torch.bool, device=x.device)
        active[nodes[W != 0]] = True
        self.n_dofs = int(2 * active.sum())

    def axis(self, xp, lp):
        inv, h = 1.0 / self.h, self.h
        lower = ((xp - lp) * inv + 1e-8).to(torch.int64)
        upper = ((xp + lp) * inv + 1e-8).to(torch.int64)
        base = (xp * inv + 1e-8).to(torch.int64)
        one = (upper == lower)
        fx = xp * inv - base
        zero = torch.zeros_like(xp)
        x0, x1, x2 = lower * h, (lower + 1) * h, (lower + 2) * h
        t0, t2 = h + lp - (xp - x0).abs(), h + lp - (xp - x2).abs()
        w = torch.stack([torch.where(one, 1.0 - fx, t0 * t0 / (4 * h * lp)),
                         torch.where(one, fx, 1.0 - ((xp - x1) ** 2 + lp * lp) / (2 * h * lp)),
                         torch.where(one, zero, t2 * t2 / (4 * h * lp))], 1)
        gw = torch.stack([torch.where(one, zero - inv, -t0 / (2 * h * lp) * torch.sign(xp - x0)),
                          torch.where(one, zero + inv, -(xp - x1) / (h * lp)),
                          torch.where(one, zero, -t2 / (2 * h * lp) * torch.sign(xp - x2))], 1)
        return lower, w, gw

    def shape(self, x, lp):
        l0, w0, g0 = self.axis(x[:, 0], lp[:, 0])
        l1, w1, g1 = self.axis(x[:, 1], lp[:, 1])
        W = (w1[:, :, None] * w0[:, None, :]).reshape(-1, 9)
        G = torch.stack([(w1[:, :, None] * g0[:, None, :]).reshape(-1, 9),
                         (g1[:, :, None] * w0[:, None, :]).reshape(-1, 9)], 2)
        a = torch.arange(9, device=x.device)
        ix = (l0[:, None] + a % 3).clamp(0, self.ncx)
        iy = (l1[:, None] + a // 3).clamp(0, self.ncy)
        return W, G, ix + iy * (self.ncx + 1)

    def stress(self, H, F, b, E):
        I = torch.eye(3, dtype=F.dtype, device=F.device)
        f = I + torch.nn.functional.pad(H, (0, 1, 0, 1))
        Fn = f @ F
        bt = f @ b @ f.transpose(-1, -2)
        J = torch.linalg.det(Fn)[..., None, None]
        E = E[..., None, None]
        lam, mu = E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))
        tr = lambda a: a.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]  # noqa: E731
        bn = bt
        if self.material == "Neo-Hookean":
            sig = mu / J * (Fn @ Fn.transpose(-1, -2) - I) + lam / J * torch.log(J) * I
        elif self.material == "Linear elasticity":
            eps = 0.5 * (Fn + Fn.transpose(-1, -2)) - I
            sig = lam * tr(eps) * I + 2 * mu * eps
        else:
            e = 0.5 * _log_sym(bt)
            tau = lam * tr(e) * I + 2 * mu * e
            if self.material == "J2":
                S = tau - tr(tau) / 3.0 * I
                nrm = torch.sqrt((S * S).sum((-2, -1)) + 1e-300)[..., None, None]
                dl = torch.clamp(nrm - KAPPA, min=0.0) / (2 * mu)
                e = e - dl * S / nrm
                tau = lam * tr(e) * I + 2 * mu * e
                bn = torch.matrix_exp(2.0 * e)
            sig = tau / J
        return f, Fn, bn, J, sig

    def local(self, du, W, G, F, b, E, ramp):
        """Residual rows [..., 9, 2] of particles from their nodal increments du [..., 9, 2]."""
        H = torch.einsum("...ak,...al->...kl", G, du)
        f, _, _, J, sig = self.stress(H, F, b, E)
        finv = torch.linalg.inv(f[..., :2, :2])
        Q = self.V0 * J * (finv.transpose(-1, -2) @ sig[..., :2, :2])
        r = -torch.einsum("...ai,...ij->...aj", G, Q)
        grav = torch.tensor([0.0, -self.g * ramp * self.rho * self.V0], dtype=du.dtype, device=du.device)
        return r + W[..., None] * grav

    def step(self, q, E, ramp):
        x, lp, F, b = q
        W, G, nodes = self.shape(x, lp)
        Wd, Gd, Fd, bd, Ed = (t.detach() for t in (W, G, F, b, E))
        dev = x.device
        # active nodes by span: a node in a particle's 3-node span whose weight may be 0 is not
        # coupled, so weights different from 0 are enough
        active = torch.zeros(self.nn, dtype=torch.bool, device=dev)
        active[nodes[Wd != 0]] = True
        free = torch.stack([active & ~self.fixed[:self.nn].bool(), active & ~self.fixed[self.nn:].bool()], 1).reshape(-1)
        idx = free.nonzero().squeeze(1)
        dof = (2 * nodes[:, :, None] + torch.arange(2, device=dev)).reshape(-1, 18)
        u = torch.zeros(2 * self.nn, dtype=torch.float64, device=dev)

        def rows(u, W, G, F, b, E):
            r = self.local(u[dof].reshape(-1, 9, 2), W, G, F, b, E, ramp)
            return torch.zeros(2 * self.nn, dtype=torch.float64, device=dev).index_add(0, dof.reshape(-1), r.reshape(-1))

        jac = torch.func.vmap(torch.func.jacfwd(lambda d, *a: self.local(d, *a, ramp)), chunk_size=4096)
        best = math.inf
        for it in range(25):
            R = rows(u, Wd, Gd, Fd, bd, Ed)[idx]
            k = jac(u[dof].reshape(-1, 9, 2), Wd, Gd, Fd, bd, Ed).reshape(-1, 18, 18)
            K = torch.zeros(4 * self.nn * self.nn, dtype=torch.float64, device=dev)
            K.index_add_(0, (dof[:, :, None] * (2 * self.nn) + dof[:, None, :]).reshape(-1), -k.reshape(-1))
            K = K.reshape(2 * self.nn, 2 * self.nn)[idx][:, idx]
            nrm = float(R.norm())
            if it > 3 and (nrm < 1e-12 or nrm > 0.5 * best):
                break
            best = min(best, nrm)
            u = u.index_add(0, idx, torch.linalg.solve(K, R))
        if E.requires_grad:
            r = rows(u, W, G, F, b, E)[idx]
            u = u.index_add(0, idx, torch.linalg.solve(K, r))
        du = u[dof].reshape(-1, 9, 2)
        _, Fn, bn, _, sig = self.stress(torch.einsum("pak,pal->pkl", G, du), F, b, E)
        xn = x + torch.einsum("pa,pal->pl", W, du)
        ln = []
        for k in range(2):
            v = self.lp0 * torch.sqrt((Fn[:, :, k] ** 2).sum(1))
            v = torch.where(xn[:, k] - v < self.lo[k], xn[:, k] - self.lo[k] - 1e-6, v)
            ln.append(torch.where(xn[:, k] + v > self.hi[k], self.hi[k] - xn[:, k] - 1e-6, v))
        return (xn, torch.stack(ln, 1), Fn, bn), sig
