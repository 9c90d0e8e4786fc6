"""The work that users have this library do, as cases that can be timed and compared.

Every case goes through the Python mirror of the C ABI (kharma_b200.block, .batch, .mesh, .ctmesh, .emhd,
.adjoint) the way a program does: the block, its geometry and its state are made once, then each pass
advances them.  The listed cases cover

  * the RK2 step of one block (`Block.step`, `DeviceDriver.step`): 2D and 3D, Cartesian modes and the
    Fishbone-Moncrief torus, WENO5 / linear MC / PPM, 1D_W and Kastaun, FP64 and the FP32-flux form,
    flux-CT and face-centred B_CT, launched one by one and replayed from a CUDA graph;
  * SMR meshes: hydro Bondi accretion through the batch, magnetized B_CT blocks;
  * extended MHD: the implicit Newton solve alone and the whole ImEx step;
  * the adjoint of a run.

A pass advances the state in place, so that passes follow one another as in a run.  `exact` restates
the RK2 step of a flux-CT block in torch, in 64 bits, from the same inputs.
"""
import dataclasses
import math

import numpy as np
import torch

from kharma_b200 import ctmesh, mesh, problems
from kharma_b200.adjoint import Run
from kharma_b200.block import Block, DeviceDriver, build_geometry
from kharma_b200.emhd import ImplicitSolver
from kharma_b200.spec import (BlockSpec, EmhdSpec, ImplicitSpec, atmosphere_spec, bondi_spec, mhdmodes_spec,
                              torus_spec)

# the bytes of one double; the FP64 operations of one face, zone or Newton iteration (counted from the
# formulas: reconstruction, 4-vectors, stress tensor, signal speeds; divergence, source, inversion, floors)
F8 = 8
FLOPS_FACE, FLOPS_ZONE, FLOPS_NEWTON = 900.0, 1500.0, 12000.0


def _step(name, problem, n1, n2, n3, recon="linear_mc", riemann="llf", precision="fp64", inverter="onedw",
          b_ct="none", graph=True):
    return {"name": name, "kind": "step", "problem": problem, "n1": n1, "n2": n2, "n3": n3, "recon": recon,
            "riemann": riemann, "precision": precision, "inverter": inverter, "b_ct": b_ct, "graph": graph}


def listed():
    return [
        # a 2D linear mode at the size of the convergence tests: launches and latency count
        _step("mode2d_weno5", "mode", 48, 40, 1, recon="weno5", graph=False),
        # the 2D torus of the parity tests
        _step("torus2d_mc", "torus", 128, 128, 1),
        # the 3D fast mode that the oracle is compared on, WENO5
        _step("mode3d_weno5", "mode", 64, 64, 64, recon="weno5"),
        # the benchmark: the FM torus at 128^3 in FP64 and in the FP32-flux form
        _step("torus3d_mc", "torus", 128, 128, 128),
        _step("torus3d_mc_fp32", "torus", 128, 128, 128, precision="fp32_flux"),
        # the reference's default inverter on an odd block, launched by a host that owns the timestep
        _step("torus3d_weno5_kastaun", "torus", 101, 75, 53, recon="weno5", inverter="kastaun", graph=False),
        # face-centred B (the default transport of multilevel meshes) on one block
        _step("torus3d_bct", "torus", 96, 64, 48, b_ct="gs05_c", graph=False),
        # SMR, hydro Bondi accretion in spherical Kerr-Schild: 25 blocks of two levels
        {"name": "smr_bondi", "kind": "smr", "nb": 25, "nx": 32, "recon": "weno5", "precision": "fp64"},
        # SMR, magnetized B_CT blocks: 15 blocks of two levels
        {"name": "smr_bct", "kind": "ctmesh", "nx": 32, "recon": "linear_mc"},
        # the implicit EMHD solve of one sub-step, as the reference runs it (forward differences)
        {"name": "emhd_newton_fd", "kind": "newton", "n1": 128, "n2": 96, "n3": 64, "jacobian": "fd"},
        # a whole ImEx step of extended MHD with the exact Jacobian
        {"name": "emhd_imex", "kind": "imex", "n1": 64, "n2": 64, "n3": 32, "recon": "linear_mc",
         "jacobian": "exact"},
        # the adjoint of two steps of the torus (forward, recompute, backward)
        {"name": "adjoint_torus", "kind": "adjoint", "n1": 64, "n2": 64, "n3": 48, "precision": "fp32_flux"},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["smr", "ctmesh", "newton", "imex", "adjoint"])
    if kind == "step":
        problem = rng.choice(["mode", "torus"])
        recon = rng.choice(["linear_mc", "linear_mc", "weno5", "weno5", "ppm", "donor_cell", "linear_vl", "ppmx",
                            "mp5", "weno5_linear"])
        if rng.random() < 0.3:
            n = (_spread(rng, 24, 400), _spread(rng, 24, 400), 1)
        else:
            n = (_spread(rng, 24, 150), _spread(rng, 16, 120), _spread(rng, 8, 96))
        precision = rng.choice(["fp64", "fp64", "fp32_flux"])
        b_ct = rng.choice(["none"] * 4 + ["bs99", "gs05_0", "gs05_c"])
        return {k: v for k, v in _step("", problem, *n, recon=recon, riemann=rng.choice(["llf", "llf", "hlle"]),
                                       precision=precision, b_ct=b_ct, inverter=rng.choice(["onedw", "kastaun"]),
                                       graph=b_ct == "none" and rng.random() < 0.5).items() if k != "name"}
    if kind == "smr":
        return {"kind": "smr", "nb": 25, "nx": 2 * _spread(rng, 8, 16), "recon": rng.choice(["linear_mc", "weno5", "ppm"]),
                "precision": rng.choice(["fp64", "fp32_flux"])}
    if kind == "ctmesh":
        return {"kind": "ctmesh", "nx": 2 * _spread(rng, 8, 16), "recon": rng.choice(["linear_mc", "weno5"])}
    if kind == "newton":
        return {"kind": "newton", "n1": _spread(rng, 24, 128), "n2": _spread(rng, 16, 96), "n3": _spread(rng, 8, 64),
                "jacobian": rng.choice(["fd", "exact"])}
    if kind == "imex":
        return {"kind": "imex", "n1": _spread(rng, 16, 64), "n2": _spread(rng, 16, 64),
                "n3": rng.choice([1, _spread(rng, 8, 32)]), "recon": rng.choice(["linear_mc", "weno5"]),
                "jacobian": rng.choice(["fd", "exact"])}
    return {"kind": "adjoint", "n1": _spread(rng, 24, 64), "n2": _spread(rng, 24, 64), "n3": _spread(rng, 8, 48),
            "precision": rng.choice(["fp64", "fp32_flux"])}


# ------------------------------------------------------------------ inputs
def _spec(case):
    kw = dict(recon=case["recon"], precision=case["precision"])
    if case["problem"] == "mode":
        s = mhdmodes_spec(case["n1"], case["n2"], case["n3"], riemann=case["riemann"], **kw)
        if case["inverter"] == "kastaun":
            s = dataclasses.replace(s, inverter="kastaun", iter_max=25, err_tol=1e-12)
    else:
        s = dataclasses.replace(torus_spec(case["n1"], case["n2"], case["n3"], inverter=case["inverter"], **kw),
                                riemann=case["riemann"])
    return dataclasses.replace(s, b_ct=case["b_ct"])


def _jitter(P, seed, amp, slots=(0, 1)):
    """rho and u times 1 + amp U(-1, 1): every zone's own value, as in a flow that has developed."""
    rng = np.random.Generator(np.random.PCG64(seed))
    for p in slots:
        P[p] *= 1.0 + amp * rng.uniform(-1.0, 1.0, size=P[p].shape)
    return P


def _light_dt(spec, geom, part=0.5):
    """A timestep that holds for any flow: `part` of 1 / sum_d (coordinate light speed / width)."""
    n3, n2, n1 = spec.shape
    sl = spec.interior[1:]
    g = np.asarray(geom["gcon"])[3, :n2, :n1][sl]
    s = 0.0
    for d in range(spec.ndim):
        b, a = g[..., 0, d + 1], g[..., 0, 0]
        disc = np.sqrt(np.maximum(b * b - a * g[..., d + 1, d + 1], 0.0))
        s = s + np.maximum(np.abs((b + disc) / a), np.abs((b - disc) / a)) / spec.dx[d]
    return float(part / np.max(s))


def _step_inputs(case, seed):
    """(spec, geometry tables, primitives, B_CT faces or None, timestep)."""
    spec = _spec(case)
    geom = build_geometry(spec)
    faces = None
    if case["problem"] == "mode":
        P = _jitter(problems.mhdmodes(spec, 3, amp=1e-2), seed, 1e-3)
        if case["b_ct"] != "none":
            faces = problems.ct_curl_faces(spec)
    elif case["b_ct"] != "none":
        P, faces = problems.fm_torus(spec, geom, seed=seed, faces=True)
    else:
        P = problems.fm_torus(spec, geom, seed=seed)
    return spec, geom, P, faces, _light_dt(spec, geom)


def _smr_mesh(case):
    if case["kind"] == "smr":
        base = dataclasses.replace(
            bondi_spec(64, 64, 64, math.log(3.0), math.log(30.0), recon=case["recon"], precision=case["precision"]),
            bc=("outflow", "outflow", "reflecting", "reflecting", "periodic", "periodic"))
        # 3 x 3 x 2 roots, the central one of the lower half refined
        return mesh.SMRMesh(base, (3, 3, 2), (case["nx"],) * 3, refine=[(1, 1, 0)])
    base = BlockSpec(nx1=32, nx2=32, nx3=32, x1min=0., x1max=1., x2min=0., x2max=1., x3min=0., x3max=1., nvar=8,
                     gam=5. / 3., recon=case["recon"], b_ct="gs05_c", driver="kharma")
    return mesh.SMRMesh(base, (2, 2, 2), (case["nx"],) * 3, refine=[(1, 1, 1)])


def _emhd_field(spec, geom, seed):
    """A smooth stratified atmosphere at rest with a radial field and a weak heat flux, each variable
    perturbed by 1e-3: the state an implicit sub-step starts from."""
    n3, n2, n1 = spec.shape
    r = np.asarray(geom["r_center"])[:, :n1]
    gcon = np.asarray(geom["gcon"])[3, :n2, :n1]
    gcov = np.asarray(geom["gcov"])[3, :n2, :n1]
    x = r / r.min()
    P = np.zeros((10,) + spec.shape)
    P[0] = (x ** -1.5)[None]
    P[1] = (0.1 * x ** -2.5)[None]
    ut = 1.0 / np.sqrt(-gcov[..., 0, 0])
    for v in range(3):
        P[2 + v] = (ut * (-1.0 / gcon[..., 0, 0]) * gcon[..., 0, 1 + v])[None]
    P[5] = (1e3 / r ** 3)[None]
    P[8] = (1e-3 * x ** -2)[None]
    P[9] = (1e-4 * x ** -2)[None]
    return _jitter(P, seed, 1e-3, (0, 1, 8, 9))


# ------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "step":
        spec, geom, P, faces, dt = _step_inputs(case, seed)
        b = Block(spec, geometry=geom)
        b.set_prims(P, faces)
        s.update(block=b, dt=dt)
        if case["graph"]:
            s.update(driver=DeviceDriver(b, dt_start=dt), stream=torch.cuda.Stream())
    elif case["kind"] == "smr":
        m = _smr_mesh(case)
        geoms, dts = {}, []

        def init(spec):
            key = (spec.x1min, spec.x2min, spec.nx1, spec.dx)
            if key not in geoms:
                geoms[key] = build_geometry(spec)
            dts.append(_light_dt(spec, geoms[key]))
            return _jitter(problems.bondi(spec, geoms[key]), seed + len(dts), 1e-3)
        s.update(batch=mesh.smr_batch(m, init), dt=None)
        s["dt"] = min(dts)
    elif case["kind"] == "ctmesh":
        m = _smr_mesh(case)
        P = [_jitter(x, seed + n, 1e-3) for n, x in enumerate(ctmesh.cut(m, ctmesh.fluid_levels(m)))]
        faces = ctmesh.cut(m, ctmesh.curl_faces_levels(m))
        s.update(mesh=ctmesh.CTMesh(m, P, faces, streams=8), dt=0.2 / (4 * case["nx"]))
    elif case["kind"] == "newton":
        spec = atmosphere_spec(case["n1"], case["n2"], case["n3"])
        geom = build_geometry(spec)
        b = Block(spec, geometry=geom)
        sol = ImplicitSolver(b, EmhdSpec(closure_type="kappa_eta", higher_order_terms=True, tau=1.0, kappa=0.1, eta=0.1))
        P = torch.tensor(_emhd_field(spec, geom, seed), device="cuda")
        U = sol.ptou(P)
        dt = 0.1
        S = torch.zeros_like(P)
        sol.add_source(P, S)
        g = torch.Generator(device="cuda").manual_seed(seed)
        S += (2 * torch.rand(P.shape, generator=g, device="cuda", dtype=torch.float64) - 1) * 1e-3 * U.abs() / dt
        # to 1e-10 of the largest conserved variable per dt, as an accuracy target is given
        tol = 1e-10 * float(U.abs().max()) / dt
        sol.set_implicit(ImplicitSpec(max_nonlinear_iter=8, rootfind_tol=tol, jacobian=case["jacobian"]))
        s.update(sol=sol, P=P, U=U, S=S, dt=dt, out=torch.empty_like(P), norm=sol.scalar_field(), fail=sol.scalar_field())
    elif case["kind"] == "imex":
        spec = dataclasses.replace(mhdmodes_spec(case["n1"], case["n2"], case["n3"], recon=case["recon"]), driver="kharma")
        geom = build_geometry(spec)
        b = Block(spec, geometry=geom)
        sol = ImplicitSolver(b, EmhdSpec(closure_type="soundspeed", higher_order_terms=False),
                             ImplicitSpec(rootfind_tol=1e-10, jacobian=case["jacobian"]))
        P0 = problems.emhdmodes(spec, amp=1e-3)
        P0 = _jitter(P0, seed, 1e-4)
        ng, n = spec.ng, spec.shape       # periodic images of the interior
        for ax, nx in ((1, spec.nx3), (2, spec.nx2), (3, spec.nx1)):
            if nx > 1:
                P0 = np.take(P0, (np.arange(nx + 2 * ng) - ng) % nx + ng, axis=ax)
        P = torch.tensor(P0, device="cuda")
        s.update(sol=sol, P=P, U=sol.ptou(P), dt=_light_dt(spec, geom, 0.2), norm=sol.scalar_field(),
                 fail=sol.scalar_field())
    else:
        spec = torus_spec(case["n1"], case["n2"], case["n3"], precision=case["precision"])
        geom = build_geometry(spec)
        b = Block(spec, geometry=geom)
        b.set_prims(problems.fm_torus(spec, geom, seed=seed))
        # the mass through the x1 faces a third of the way out
        w = np.zeros(spec.shape)
        k, j, _ = spec.interior
        w[k, j, spec.ng + spec.nx1 // 3] = spec.dx[1] * spec.dx[2]
        s.update(block=b, run=Run(b, [_light_dt(spec, geom)] * 2, weight=w, checkpoint_every=2))
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "step":
        b = s["block"]
        if "driver" in s:
            with torch.cuda.stream(s["stream"]):
                s["driver"].step()
        else:
            b.step(s["dt"])
        out = {"P": b.P, "U": b.U, "pflag": b.pflag, "fflag": b.fflag}
        if b.ct:
            out["Bf"] = b.Bf
        return out
    if kind == "smr":
        s["batch"].step_graph(s["dt"])
        return {"P": [b.P for b in s["batch"].blocks], "U": [b.U for b in s["batch"].blocks]}
    if kind == "ctmesh":
        s["mesh"].step_graph(s["dt"])
        return {"P": [b.P for b in s["mesh"].blocks], "U": [b.U for b in s["mesh"].blocks],
                "Bf": [b.Bf for b in s["mesh"].blocks]}
    if kind == "newton":
        s["out"].copy_(s["P"])                       # the guess: the state at the start of the sub-step
        s["fail"].zero_()
        s["sol"].step(s["P"], s["U"], s["P"], s["S"], s["out"], s["norm"], s["fail"], s["dt"])
        return {"P": s["out"], "fail": s["fail"]}
    if kind == "imex":
        s["fail"].zero_()
        s["sol"].imex_step(s["P"], s["U"], s["dt"], s["norm"], s["fail"])
        return {"P": s["P"], "U": s["U"], "fail": s["fail"]}
    J = s["run"].forward()
    Pbar, Ubar = s["run"].adjoint()
    return {"J": J, "Pbar": Pbar, "Ubar": Ubar}


# ------------------------------------------------------------------ work, tolerance
def work(case):
    """Each state variable read and written once (P and U, faces, flags); the FP64 (or FP32) operations
    of the formulas, without any recomputation."""
    k = case["kind"]
    if k == "step":
        z = case["n1"] * case["n2"] * case["n3"]
        nd = 2 + (case["n3"] > 1)
        return {"bytes": z * (4 * 8 * F8 + 8 + (6 * F8 if case["b_ct"] != "none" else 0)),
                "flops": z * 2 * (nd * FLOPS_FACE + FLOPS_ZONE)}
    if k == "smr":
        z = case["nb"] * case["nx"] ** 3
        return {"bytes": z * (4 * 5 * F8 + 8), "flops": z * 2 * (3 * 500.0 + 900.0)}
    if k == "ctmesh":
        z = 15 * case["nx"] ** 3
        return {"bytes": z * (4 * 8 * F8 + 8 + 6 * F8), "flops": z * 2 * (3 * FLOPS_FACE + FLOPS_ZONE)}
    z = case["n1"] * case["n2"] * case["n3"]
    if k == "newton":
        return {"bytes": z * F8 * (4 * 10 + 7 + 4), "flops": z * 2 * FLOPS_NEWTON}
    if k == "imex":
        nd = 2 + (case["n3"] > 1)
        return {"bytes": z * F8 * (4 * 10 + 4), "flops": z * 2 * (nd * 1.5 * FLOPS_FACE + FLOPS_ZONE + 2 * FLOPS_NEWTON)}
    # two steps forward, recomputed, and their adjoint at a few times a step's cost
    return {"bytes": z * F8 * 4 * 8 * 6, "flops": z * 2 * 6 * 2 * (3 * FLOPS_FACE + FLOPS_ZONE)}


def tolerance(case):
    """About four times the difference that contracting multiplies and adds throughout makes (FP64 paths) or
    that the FP32 fluxes have against `exact` (the FP32-flux form): the inversion stops at 1e-8 of its
    unknown, so a rounding difference reaches the primitives at 1e-12; the adjoint carries it through the
    derivative of limiters and fixups."""
    k = case["kind"]
    fp32 = case.get("precision") == "fp32_flux"
    if k == "adjoint":
        rel, most = (1e-6, 7e-4) if fp32 else (5e-9, 1e-6)
    elif fp32:
        rel, most = 1e-6, 2e-4
    elif k == "step":
        rel, most = 6e-12, 2.5e-9
    elif k == "imex":
        rel, most = 1e-11, 1e-9
    elif k == "newton":
        rel, most = 2e-13, 4e-12
    else:
        rel, most = 4e-13, 4e-11
    return {"rel": rel, "max": most, "differ": 1e-5}


# ------------------------------------------------------------------ the step in 64 bits
class _Ref:
    """One RK2 step of a flux-CT block (recon linear_mc, weno5, ppm or donor_cell) in torch, 64 bits, on
    whole arrays: values outside the range a formula is valid on are computed and not used."""

    def __init__(self, spec, geom):
        self.s = spec
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        n3, n2, n1 = spec.shape
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)
        cut = lambda a: t(np.asarray(a)[:4, :n2, :n1])
        self.gcov, self.gcon, self.gdet = cut(geom["gcov"]), cut(geom["gcon"]), cut(geom["gdet"])
        self.conn = t(geom["gdet_conn"])
        r = t(np.asarray(geom["r_center"])[:n2, :n1])
        f = spec.floors
        if spec.spherical:
            sc = 1.0 / torch.sqrt(r ** 3)
            self.rho_fl = torch.clamp(f.rho_min_geom * sc, min=f.rho_min_const)
            self.u_fl = torch.clamp(f.u_min_geom * sc ** spec.gam, min=f.u_min_const)
        else:
            self.rho_fl, self.u_fl = torch.full_like(r, f.rho_min_const), torch.full_like(r, f.u_min_const)
        self.ng = spec.ng
        self.lo = [spec.ng if n > 1 else 0 for n in (spec.nx3, spec.nx2, spec.nx1)]
        self.hi = [l + n for l, n in zip(self.lo, (spec.nx3, spec.nx2, spec.nx1))]

    # shift along direction d (1..3): the value `m` zones further
    def at(self, x, d, m):
        return torch.roll(x, -m, dims=x.dim() - d)

    def vecs(self, P, loc):
        g, h = self.gcov[loc], self.gcon[loc]
        u, B = P[2:5], P[5:8]
        q = sum(g[..., a + 1, b + 1] * u[a] * u[b] for a in range(3) for b in range(3))
        gam, al = torch.sqrt(1 + q), 1 / torch.sqrt(-h[..., 0, 0])
        uc = [gam / al] + [u[v] - gam * al * h[..., 0, v + 1] for v in range(3)]
        low = lambda c: [sum(g[..., m, n] * c[n] for n in range(4)) for m in range(4)]
        ud = low(uc)
        b0 = sum(B[v] * ud[v + 1] for v in range(3))
        bc = [b0] + [(B[v] + b0 * uc[v + 1]) / uc[0] for v in range(3)]
        return uc, ud, bc, low(bc)

    def flux(self, P, V, loc, d):
        uc, ud, bc, bd = V
        g = self.s.gam
        bsq = sum(bc[m] * bd[m] for m in range(4))
        pg = (g - 1) * P[1]
        eta, pt = pg + P[0] + P[1] + bsq, pg + 0.5 * bsq
        T = [eta * uc[d] * ud[m] + (pt if m == d else 0) - bc[d] * bd[m] for m in range(4)]
        D = P[0] * uc[d]
        B = [P[5 + v] if d == 0 else bc[v + 1] * uc[d] - bc[d] * uc[v + 1] for v in range(3)]
        return torch.stack([D, T[0] + D, T[1], T[2], T[3]] + B) * self.gdet[loc]

    def speeds(self, P, V, loc, d):
        uc, _, bc, bd = V
        g, h = self.s.gam, self.gcon[loc]
        ef = P[0] + g * P[1]
        bsq = sum(bc[m] * bd[m] for m in range(4))
        cs, va = g * (g - 1) * P[1] / ef, bsq / (bsq + ef)
        c = cs + va - cs * va
        A = uc[0] ** 2 - (h[..., 0, 0] + uc[0] ** 2) * c
        B = 2 * (uc[d] * uc[0] - (h[..., 0, d] + uc[d] * uc[0]) * c)
        C = uc[d] ** 2 - (h[..., d, d] + uc[d] ** 2) * c
        q = torch.sqrt(torch.clamp(B * B - 4 * A * C, min=0))
        return (B - q) / (2 * A), (B + q) / (2 * A)

    def recon(self, P, d):
        """Left and right face values of every zone along d."""
        x = [self.at(P, d, m) for m in (-2, -1, 0, 1, 2)]
        k = self.s.recon
        if k == "donor_cell":
            return x[2], x[2]
        if k == "linear_mc":
            dm, dp = x[2] - x[1], x[3] - x[2]
            r = torch.where(dp.abs() > 0, dm / dp, torch.full_like(dp, 2.0))
            s = torch.clamp(torch.minimum(2 * r, 0.5 * (1 + r)), 0, 2) * dp
            return x[2] - 0.5 * s, x[2] + 0.5 * s
        if k == "weno5":
            def side(a, b, c, e, f):
                d0 = (1e-26 + 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2) ** 2
                d1 = (1e-26 + 13 / 12 * (b - 2 * c + e) ** 2 + 0.25 * (e - b) ** 2) ** 2
                d2 = (1e-26 + 13 / 12 * (c - 2 * e + f) ** 2 + 0.25 * (f - 4 * e + 3 * c) ** 2) ** 2
                w = [1 / 16 / d0, 5 / 8 / d1, 5 / 16 / d2]
                W = w[0] + w[1] + w[2]
                return ((3 / 8 * a - 5 / 4 * b + 15 / 8 * c) * (w[0] / W) + (-1 / 8 * b + 3 / 4 * c + 3 / 8 * e) * (w[1] / W)
                        + (3 / 8 * c + 3 / 4 * e - 1 / 8 * f) * (w[2] / W))
            return side(*x[::-1]), side(*x)
        if k == "ppm":
            mn, mx = torch.minimum, torch.maximum
            l = (7 * (x[2] + x[1]) - (x[0] + x[3])) / 12
            r = (7 * (x[2] + x[3]) - (x[1] + x[4])) / 12
            l = mn(mx(l, mn(x[2], x[1])), mx(x[2], x[1]))
            r = mn(mx(r, mn(x[2], x[3])), mx(x[2], x[3]))
            qc, qd = r - x[2], l - x[2]
            flat = qc * qd >= 0
            r2 = torch.where(qc.abs() >= 2 * qd.abs(), x[2] - 2 * qd, r)
            l2 = torch.where(qd.abs() >= 2 * qc.abs(), x[2] - 2 * qc, l)
            return torch.where(flat, x[2], l2), torch.where(flat, x[2], r2)
        return None

    def faces(self, P):
        """Face fluxes and ctop per direction (face i between zones i - 1 and i)."""
        F = []
        for d in range(1, self.s.ndim + 1):
            Rr, R = self.recon(P, d)
            L, loc = self.at(R, d, -1), d - 1                # left state: right face value of the zone below
            VL, VR = self.vecs(L, loc), self.vecs(Rr, loc)
            sL, sR = self.speeds(L, VL, loc, d), self.speeds(Rr, VR, loc, d)
            up = torch.clamp(torch.maximum(torch.maximum(*sL), torch.maximum(*sR)), min=0)
            dn = -torch.clamp(torch.minimum(torch.minimum(*sL), torch.minimum(*sR)), max=0)
            fl, fr = self.flux(L, VL, loc, d), self.flux(Rr, VR, loc, d)
            ul, ur = self.flux(L, VL, loc, 0), self.flux(Rr, VR, loc, 0)
            if self.s.riemann == "llf":
                F.append(0.5 * (fl + fr - torch.maximum(up, dn) * (ur - ul)))
            else:
                F.append((up * fl + dn * fr - up * dn * (ur - ul)) / (up + dn))
        return F

    def fix(self, F):
        s = self.s
        if s.spherical and s.ndim > 1 and s.bc[2] == "reflecting":
            j0, j1 = self.lo[1], self.hi[1]
            for j, a, b in ((j0, j0 - 1, j0), (j1, j1, j1 - 1)):
                if s.fix_polar_flux:
                    F[1][5][:, j], F[1][7][:, j] = 0.0, 0.0
                    F[0][6][:, a] = -F[0][6][:, b]
                    if s.ndim > 2:
                        F[2][6][:, a] = -F[2][6][:, b]
                if s.zero_polar_flux:
                    F[1][:, :, j] = 0.0
        if s.check_inflow_inner_x1:
            F[0][0][..., self.lo[2]].clamp_(max=0)
        if s.check_inflow_outer_x1:
            F[0][0][..., self.hi[2]].clamp_(min=0)
        return F

    def flux_ct(self, F):
        s, at = self.s, self.at
        e3 = 0.25 * (F[0][6] + at(F[0][6], 2, -1) - F[1][5] - at(F[1][5], 1, -1))
        F[0][5], F[0][6] = 0.0, 0.5 * (e3 + at(e3, 2, 1))
        new = {(1, 5): -0.5 * (e3 + at(e3, 1, 1)), (1, 6): torch.zeros_like(e3)}
        if s.ndim > 2:
            e1 = 0.25 * (F[1][7] + at(F[1][7], 3, -1) - F[2][6] - at(F[2][6], 2, -1))
            e2 = 0.25 * (F[2][5] + at(F[2][5], 1, -1) - F[0][7] - at(F[0][7], 3, -1))
            F[0][7] = -0.5 * (e2 + at(e2, 3, 1))
            new[(1, 7)] = 0.5 * (e1 + at(e1, 3, 1))
            new[(2, 5)], new[(2, 6)] = 0.5 * (e2 + at(e2, 1, 1)), -0.5 * (e1 + at(e1, 2, 1))
            new[(2, 7)] = torch.zeros_like(e1)
        for (d, p), v in new.items():
            F[d][p] = v
        if s.zero_polar_flux and s.bc[2] == "reflecting":
            F[1][5:8, :, self.lo[1]] = 0.0
            F[1][5:8, :, self.hi[1]] = 0.0
        return F

    def invert(self, U, P):
        """Primitives from U (P: the guess), 1D_W or Kastaun; (P, failed)."""
        s, g, h = self.s, self.gcov[3], self.gcon[3]
        al = 1 / torch.sqrt(-h[..., 0, 0])
        k = al / self.gdet[3]
        D, B = U[0] * k, [U[5 + v] * k for v in range(3)]
        Q = [(U[1] - U[0]) * k] + [U[2 + v] * k for v in range(3)]
        new = P.clone()
        if s.inverter == "kastaun":
            return self.kastaun(U, new, D, B, Q, al)
        Qu = [sum(h[..., m, n] * Q[n] for n in range(4)) for m in range(4)]
        nu = [-h[..., m, 0] * al for m in range(4)]
        Bd = [sum(g[..., m, v + 1] * B[v] for v in range(3)) for m in range(4)]
        Bsq = sum(B[v] * Bd[v + 1] for v in range(3))
        QB = sum(B[v] * Q[v + 1] for v in range(3))
        Qn = -al * Qu[0]
        Qt = sum(Qu[m] * Q[m] for m in range(4)) + Qn * Qn
        Ep = -Qn - D
        bad = U[0] <= 0

        def lor(Wp):
            W = Wp + D
            WB = W + Bsq
            u2 = -((W + WB) * QB ** 2 + W ** 2 * Qt) / (QB ** 2 * (W + WB) + W ** 2 * (Qt - WB ** 2))
            return torch.where((u2 < -1e-15) | (u2 > 1e7), torch.full_like(u2, -1.0), torch.sqrt(1 + u2.abs()))

        def err(Wp):
            W, ga = Wp + D, lor(Wp)
            p = (W / ga ** 2 - D / ga) * (s.gam - 1) / s.gam
            return -Ep + Wp - p + 0.5 * Bsq + 0.5 * (Bsq * Qt - QB ** 2) / (Bsq + W) ** 2
        u = P[2:5]
        ga = torch.sqrt(1 + sum(g[..., a + 1, b + 1] * u[a] * u[b] for a in range(3) for b in range(3)))
        W = (P[0] + s.gam * P[1]) * ga ** 2 - P[0] * ga
        e = err(W)
        Wm = (1 - 1e-5) * W
        hh = W - Wm
        em, ep = err(Wm), err(W + hh)
        d1, d2 = (ep - em) / (W + hh - Wm), (ep - 2 * e + em) / (hh * hh)
        f = torch.clamp(0.5 * e * d2 / (d1 * d1), -0.3, 0.3)
        dW = torch.minimum(torch.maximum(-e / d1 / (1 - f), -0.5 * W), 2 * W)
        W1, e1 = W, e
        W = W + dW
        e = err(W)
        done = torch.zeros_like(bad)
        for _ in range(s.iter_max):
            dW = torch.minimum(torch.maximum((W1 - W) * e / (e - e1), -0.5 * W), 2 * W)
            Wn = W + dW
            en = err(Wn)
            stop = ((dW / Wn).abs() < s.err_tol) | ((en / Wn).abs() < s.err_tol)
            W1, e1, W, e = (torch.where(done, a, b) for a, b in ((W1, W), (e1, e), (W, Wn), (e, en)))
            done = done | stop
        bad = bad | ~done
        ga, w = lor(W), W + D
        bad = bad | (ga < 1)
        rho, w2 = D / ga, w / ga ** 2
        uu = w2 - rho - (w2 - rho) * (s.gam - 1) / s.gam
        bad = bad | (rho < 0) | (uu < 0)
        for p, v in enumerate([rho, uu] + [ga / (w + Bsq) * (Qu[m + 1] + nu[m + 1] * Qn + QB * B[m] / w) for m in range(3)]):
            new[p] = torch.where(bad, P[p], v)
        return new, bad

    def kastaun(self, U, new, D, B, Q, al):
        s, g, h, f = self.s, self.gcov[3], self.gcon[3], self.s.floors
        Df = torch.clamp(D, min=f.rho_min_const)
        q = (-sum(Q[m] * -al * h[..., m, 0] for m in range(4)) - D) / D
        r = [U[2 + v] / U[0] for v in range(3)]
        ru = [sum((h[..., a + 1, b + 1] - h[..., 0, a + 1] * h[..., 0, b + 1] / h[..., 0, 0]) * r[b] for b in range(3))
              for a in range(3)]
        rsq = sum(ru[a] * r[a] for a in range(3))
        b = [x / torch.sqrt(Df) for x in B]
        br = sum(b[a] * r[a] for a in range(3))
        bsq = torch.clamp(sum(g[..., a + 1, c + 1] * b[a] * b[c] for a in range(3) for c in range(3)), min=0)
        rb = br * br
        v0 = torch.clamp(rsq / (1 + rsq), max=1 - 1 / f.gamma_max ** 2)
        ef = f.u_min_const / Df

        def parts(mu):
            x = 1 / (1 + mu * bsq)
            rbar = x * (x * rsq + mu * (1 + x) * rb)
            qb = q - 0.5 * (bsq + (mu * x) ** 2 * (bsq * rsq - rb))
            v = torch.minimum(mu * mu * rbar, v0)
            W = 1 / torch.sqrt(1 - v)
            rho = torch.clamp(D / W, min=f.rho_min_const)
            e = W * (qb - mu * rbar) + v * W * W / (1 + W)
            return x, rbar, qb, W, rho, torch.minimum(torch.maximum(e, ef), torch.full_like(e, f.u_over_rho_max))

        def master(mu):
            x, rbar, qb, W, rho, e = parts(mu)
            p = (s.gam - 1) * rho * e
            a = p / (rho * (1 + e))
            return mu - 1 / (torch.maximum((1 + a) * (1 + e) / W, (1 + a) * (1 + qb - mu * rbar)) + mu * rbar)

        def aux(mu):
            x = 1 / (1 + mu * bsq)
            return mu * torch.sqrt(1 + x * (x * rsq + mu * (1 + x) * rb)) - 1

        def root(fn, hi):                          # bisection to the last bits; master and aux rise through it
            lo = torch.zeros_like(hi)
            for _ in range(70):
                m = 0.5 * (lo + hi)
                below = fn(m) < 0
                lo, hi = torch.where(below, m, lo), torch.where(below, hi, m)
            return 0.5 * (lo + hi)
        mu = root(master, root(aux, torch.ones_like(D)) * (1 + 1e-15))
        x, _, _, W, rho, e = parts(mu)
        for p, v in enumerate([rho, e * rho] + [W * mu * x * (ru[a] + mu * br * b[a]) for a in range(3)]):
            new[p] = v
        return new, torch.zeros_like(D, dtype=torch.bool)

    def floors(self, P):
        s, g, h, f = self.s, self.gcov[3], self.gcon[3], self.s.floors
        V = self.vecs(P, 3)
        uc, ud, bc, bd = V
        bsq = sum(bc[m] * bd[m] for m in range(4))
        uf = torch.maximum(self.u_fl + 0 * bsq, bsq / f.bsq_over_u_max)
        rf = torch.maximum(torch.maximum(self.rho_fl + 0 * bsq, bsq / f.bsq_over_rho_max),
                           torch.maximum(P[1], uf) / f.u_over_rho_max)
        lor = lambda u: torch.sqrt(1 + sum(g[..., a + 1, b + 1] * u[a] * u[b] for a in range(3) for b in range(3)))
        hit = (rf > P[0]) | (uf > P[1]) | (lor(P[2:5]) > f.gamma_max) | ((s.gam - 1) * P[1] / P[0] ** s.gam > f.ktot_max)
        # drift frame
        w = torch.clamp(P[0] + s.gam * P[1], min=1e-20)
        B = [P[5 + v] for v in range(3)]
        Bd = [sum(g[..., m, v + 1] * B[v] for v in range(3)) for m in range(4)]
        Bm = torch.sqrt(torch.clamp(sum(B[v] * Bd[v + 1] for v in range(3)), min=1e-20))
        QB = sum(B[v] * (w * uc[0] * ud[v + 1]) for v in range(3))
        vp = QB / (Bm * w * uc[0] ** 2)
        dr0 = 1 / torch.sqrt(1 / uc[0] ** 2 + vp ** 2)
        dr = [dr0] + [uc[v + 1] * (dr0 / uc[0]) - vp * B[v] * dr0 / Bm for v in range(3)]
        rho, u = torch.maximum(P[0], rf), torch.maximum(P[1], uf)
        x = 2 * QB / (Bm * (rho + s.gam * u) * dr0)
        vp = x / (1 + torch.sqrt(1 + x * x)) / dr0
        uc0 = 1 / torch.sqrt(1 / dr0 ** 2 - vp ** 2)
        N = [rho, u] + [dr[v + 1] * (uc0 / dr0) + vp * B[v] * uc0 / Bm - h[..., 0, v + 1] / h[..., 0, 0] * uc0 for v in range(3)]
        ga = lor(N[2:5])
        sc = torch.where(ga > f.gamma_max, torch.sqrt((f.gamma_max ** 2 - 1) / (ga ** 2 - 1)), torch.ones_like(ga))
        N[2:5] = [v * sc for v in N[2:5]]
        kt = (s.gam - 1) * N[1] / N[0] ** s.gam
        N[1] = torch.where(kt > f.ktot_max, f.ktot_max / kt * N[1], N[1])
        out = P.clone()
        for p in range(5):
            out[p] = torch.where(hit, N[p], P[p])
        return out

    def p_to_u(self, P):
        return self.flux(P, self.vecs(P, 3), 3, 0)

    def fixup(self, P, bad):
        s = self.s
        inside = torch.zeros_like(bad)
        inside[self.box()] = True
        bad = bad & inside
        if not bool(bad.any()):
            return P
        num, den = torch.zeros_like(P[:5]), torch.zeros_like(P[0])
        k, j, i = torch.nonzero(bad, as_tuple=True)
        if s.fix_average_neighbors:
            for dk in (-1, 0, 1):
                for dj in (-1, 0, 1):
                    for di in (-1, 0, 1):
                        x, ok = [k + dk, j + dj, i + di], torch.ones_like(k, dtype=torch.bool)
                        for a, bc in ((0, s.bc[4]), (1, s.bc[2]), (2, s.bc[0])):
                            n = self.hi[a] - self.lo[a]
                            if bc == "periodic" and n > 1:
                                x[a] = (x[a] - self.lo[a]) % n + self.lo[a]
                            ok &= (x[a] >= self.lo[a]) & (x[a] < self.hi[a])
                        x = [torch.where(ok, v, torch.full_like(v, l)) for v, l in zip(x, self.lo)]
                        ok &= ~bad[x[0], x[1], x[2]]
                        w = ok.double() / (abs(dk) + abs(dj) + abs(di) + 1)
                        den[k, j, i] += w
                        num[:, k, j, i] += w * P[:5, x[0], x[1], x[2]]
        mean = torch.where(den < 1e-10, torch.zeros_like(num), num / den.clamp(min=1e-300))
        mean[0], mean[1] = torch.maximum(mean[0], self.rho_fl + 0 * den), torch.maximum(mean[1], self.u_fl + 0 * den)
        P = P.clone()
        P[:5] = torch.where(bad, mean, P[:5])
        return P

    def box(self):
        return tuple(slice(a, b) for a, b in zip(self.lo, self.hi))

    def ghosts(self, P, U):
        """Boundary conditions on P (fluid) and U (field), then P_B, U = U(P) there; in place."""
        s, ng = self.s, self.ng
        (k0, j0, i0), (k1, j1, i1) = self.lo, self.hi
        kk = slice(k0, k1)

        def face(inner, axis, rows):
            a, b = (self.lo[axis], self.hi[axis])
            kind = s.bc[2 * (2 - axis) + (0 if inner else 1)]
            dst = list(range(0, a)) if inner else list(range(b, b + ng))
            ref = a if inner else b - 1
            src = [ref] * ng if kind == "outflow" else [2 * ref + (-1 if inner else 1) - x for x in dst]
            ix = lambda m: (kk, rows, m) if axis == 2 else (kk, m, rows)
            for d, c in zip(dst, src):
                for p in range(5):
                    P[p][ix(d)] = P[p][ix(c)] * (-1.0 if kind == "reflecting" and p == (4 - axis) else 1.0)
                for v in range(3):
                    U[5 + v][ix(d)] = U[5 + v][ix(c)] * (-1.0 if kind == "reflecting" and v == 2 - axis else 1.0)
                if axis == 2 and (s.check_inflow_inner_x1 if inner else s.check_inflow_outer_x1):
                    self.inflow(P, kk, rows, d, inner)
        phys = s.bc[0] != "periodic" or (s.ndim > 1 and s.bc[2] != "periodic")
        if s.bc[0] != "periodic":
            face(True, 2, slice(j0, j1))
            face(False, 2, slice(j0, j1))
        if s.ndim > 1 and s.bc[2] != "periodic":
            face(True, 1, slice(None))
            face(False, 1, slice(None))
            if s.fix_corner_inner and s.bc[0] != "periodic":
                face(True, 2, slice(None))
        if phys:
            ghost = torch.ones(P.shape[1:], dtype=torch.bool, device=self.dev)
            ghost[self.box()] = False
            for v in range(3):
                P[5 + v] = torch.where(ghost, U[5 + v] / self.gdet[3], P[5 + v])
            U.copy_(torch.where(ghost, self.p_to_u(P), U))
        per = lambda a, bc, n: [(x - a) % n + a if bc == "periodic" and n > 1 else x for x in range(n + 2 * a)]
        ix = [torch.tensor(per(l, bc, h - l), device=self.dev) for l, h, bc in zip(self.lo, self.hi, (s.bc[4], s.bc[2], s.bc[0]))]
        for X in (P, U):
            X.copy_(X[:, ix[0]][:, :, ix[1]][:, :, :, ix[2]])

    def inflow(self, P, kk, rows, i, inner):
        g, h = self.gcov[3][rows, i], self.gcon[3][rows, i]
        u = [P[2 + v][kk, rows, i] for v in range(3)]
        dot = lambda a: sum(g[..., x + 1, y + 1] * a[x] * a[y] for x in range(3) for y in range(3))
        ga, al = torch.sqrt(1 + dot(u)), 1 / torch.sqrt(-h[..., 0, 0])
        u1 = u[0] - ga * al * h[..., 0, 1]
        enter = u1 > 0 if inner else u1 < 0
        v = [al * h[..., 0, 1] + 0 * ga, u[1] / ga, u[2] / ga]
        gn = 1 / torch.sqrt(1 - dot(v))
        for p in range(3):
            P[2 + p][kk, rows, i] = torch.where(enter, v[p] * gn, u[p])

    def stage(self, P, U, U0, g0, g1, dt):
        s, b = self.s, self.box()
        F = self.flux_ct(self.fix(self.faces(P)))
        div = sum((self.at(F[d], d + 1, 1) - F[d]) / s.dx[d] for d in range(s.ndim))
        new = g0 * U + g1 * U0 - dt * div
        if not s.cart_minkowski:
            V = self.vecs(P, 3)
            for m in range(4):
                T = self.flux_row(P, V, m)
                for l in range(4):
                    new[1 + l] += dt * sum(T[n] * self.conn[..., n, l, m] for n in range(4))
        Pn, bad = self.invert(new, P)
        for v in range(3):
            Pn[5 + v] = new[5 + v] / self.gdet[3]
        if s.floors_on:
            Pn = self.floors(Pn)
        Pn = self.fixup(Pn, bad)
        Po, Uo = P.clone(), U.clone()
        ix = (slice(None),) + b
        Po[ix] = Pn[ix]
        Uo[ix] = self.p_to_u(Pn)[ix]
        self.ghosts(Po, Uo)
        return Po, Uo

    def flux_row(self, P, V, m):
        uc, ud, bc, bd = V
        bsq = sum(bc[n] * bd[n] for n in range(4))
        pg = (self.s.gam - 1) * P[1]
        return [(pg + P[0] + P[1] + bsq) * uc[m] * ud[n] + (pg + 0.5 * bsq if m == n else 0) - bc[m] * bd[n] for n in range(4)]

    def step(self, P0, dt):
        P = torch.as_tensor(P0, dtype=torch.float64, device=self.dev).clone()
        U = self.p_to_u(P)
        self.ghosts(P, U)
        U = self.p_to_u(P)
        P1, U1 = self.stage(P, U, U, 1.0, 0.0, dt)
        return self.stage(P1, U1, U, 0.5, 0.5, 0.5 * dt)


def exact(case, seed):
    """P and U after the first step, for flux-CT blocks with the reconstructions _Ref has; the other
    paths (face-centred B, meshes, EMHD, the adjoint) have no short restatement."""
    if case["kind"] != "step" or case["b_ct"] != "none" or case["recon"] not in ("linear_mc", "weno5", "ppm", "donor_cell"):
        return None
    spec, geom, P, _, dt = _step_inputs(case, seed)
    P, U = _Ref(spec, geom).step(P, dt)
    return {"P": P, "U": U, "pflag": None, "fflag": None}
