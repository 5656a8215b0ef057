"""The work a user of this library has it do, as cases that can be timed and compared.

Every case advances one flow case (or one batch of them) through the package's
public calls: ``JoeGpu.runBackwardEuler`` + ``get_state`` (the state stays on the
device between calls), ``JoeGpu.step_host`` (the state lives in page-locked host
arrays and is stepped in place) or ``JoeGpuBatch.runBackwardEulerCases`` (many
cases in one handle).  The meshes, fluids and solver settings are those of
``myjoe_b200.case``, the benchmark and the batch driver; the CFL ramps stop at
moderate values so that a case can be marched on for thousands of steps.  The
initial state is the free stream with a smooth perturbation drawn from the seed.

``exact`` is the same iteration in plain 64-bit torch for the inviscid HLLC
cases with point relaxation; the laminar Roe, turbulence and batched cases have
no independent 64-bit value here.
"""
import dataclasses
import functools
import math
import types

import numpy as np
import torch

from myjoe_b200 import batch, case as jcase, geometry, solver

SGS_LAG = 4   # the serving and batching drivers' lagged Jacobian


def listed():
    return [
        # the smallest call: one step at a time on 5,000 cells, the residual read after each step as
        # the reference's loop does; launch latency counts
        dict(name="bump_5k_one_step", kind="bump", nx=100, ny=25, nz=2, flux="HLLC", order2=True, solver="JACOBI",
             sweeps=10, mixed=False, lag=1, renumber=0, steps=1, call="march"),
        # the inviscid channel bump at 8,192 cells, multicolour Gauss-Seidel: an ordinary small case
        dict(name="bump_8k_sgs", kind="bump", nx=64, ny=32, nz=4, flux="HLLC", order2=True, solver="SGS",
             sweeps=10, mixed=False, lag=1, renumber=0, steps=10, call="march"),
        # odd and ragged sizes, another flux (AUSM; implicit side HLLC), the serving form's mixed precision
        dict(name="bump_31k_odd_mixed", kind="bump", nx=157, ny=67, nz=3, flux="AUSM", order2=True, solver="SGS",
             sweeps=7, mixed=True, lag=SGS_LAG, renumber=2, steps=11, call="march"),
        # the benchmark's laminar plate, device-resident state
        dict(name="plate_49k_march", kind="plate", nx=256, ny=96, nz=2, solver="JACOBI", sweeps=10, mixed=False,
             lag=1, renumber=0, steps=20, call="march"),
        # the benchmark's end-to-end call: host-resident state, one step a call
        dict(name="plate_49k_host", kind="plate", nx=256, ny=96, nz=2, solver="JACOBI", sweeps=10, mixed=False,
             lag=1, renumber=0, steps=1, call="host"),
        # the reference's own linear solver on the plate (restarted from the initial state each call,
        # so that every call does the same iterations)
        dict(name="plate_49k_bcgstab", kind="plate", nx=256, ny=96, nz=2, solver="BCGSTAB", sweeps=10, mixed=False,
             lag=1, renumber=0, steps=2, call="restart"),
        # a large case of the serving stream: mixed precision, lagged Jacobian, colour-grouped order
        dict(name="bump_250k_mixed", kind="bump", nx=500, ny=250, nz=2, flux="HLLC", order2=True, solver="SGS",
             sweeps=10, mixed=True, lag=SGS_LAG, renumber=2, steps=16, call="host"),
        # the memory-bound end of the range: the benchmark's 1.96M-cell bump
        dict(name="bump_2m_fp64", kind="bump", nx=1400, ny=700, nz=2, flux="HLLC", order2=True, solver="JACOBI",
             sweeps=10, mixed=False, lag=1, renumber=0, steps=4, call="host"),
        # Spalart-Allmaras on the shuffled prism/hexahedron mesh, line relaxation, plain and mixed form
        dict(name="sa_100k_line_fp64", kind="sa", nx=256, ny=80, nz=4, n_prism=18, stretch=1.1, solver="LINE",
             sweeps=10, mixed=False, renumber=3, steps=5, call="march"),
        dict(name="sa_100k_line_mixed", kind="sa", nx=256, ny=80, nz=4, n_prism=18, stretch=1.1, solver="LINE",
             sweeps=10, mixed=True, renumber=3, steps=5, call="march"),
        # the batching form: inviscid cases of uneven size in one handle
        dict(name="batch_24_bumps", kind="batch", model="EULER", cases=24, lo=4000, hi=40000, pick=5, solver="SGS",
             sweeps=10, mixed=True, lag=SGS_LAG, renumber=2, steps=10),
        # the batching form: Menter SST cases, line relaxation
        dict(name="batch_8_sst", kind="batch", model="SST", cases=8, lo=5000, hi=20000, pick=3, solver="LINE",
             sweeps=10, mixed=True, lag=1, renumber=2, steps=6),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["bump", "bump", "bump", "plate", "sa", "batch"])
    mixed = rng.random() < 0.5
    if kind == "batch":
        if rng.random() < 0.6:
            return dict(kind="batch", model="EULER", cases=rng.randint(3, 24), lo=4000, hi=40000,
                        pick=rng.randint(10, 10 ** 6), solver=rng.choice(["SGS", "JACOBI"]),
                        sweeps=rng.randint(4, 12), mixed=mixed, lag=rng.choice([1, SGS_LAG]),
                        renumber=rng.choice([0, 2]), steps=rng.randint(4, 10))
        return dict(kind="batch", model="SST", cases=rng.randint(2, 8), lo=4000, hi=20000,
                    pick=rng.randint(10, 10 ** 6), solver=rng.choice(["LINE", "SGS"]), sweeps=rng.randint(4, 10),
                    mixed=mixed, lag=1, renumber=rng.choice([0, 2]), steps=rng.randint(3, 6))
    if kind == "sa":
        nx = int(_log_uniform(rng, 60, 240))
        ny = rng.randint(40, 80)
        return dict(kind="sa", nx=nx, ny=ny, nz=rng.randint(2, 4), n_prism=rng.choice([0, ny // 4]), stretch=1.1,
                    solver=rng.choice(["LINE", "LINE", "SGS"]), sweeps=rng.randint(4, 10), mixed=mixed,
                    renumber=rng.choice([1, 3]), steps=rng.randint(3, 6), call="march")
    if kind == "plate":
        nx = int(_log_uniform(rng, 60, 500))
        return dict(kind="plate", nx=nx, ny=rng.randint(48, 100), nz=rng.randint(1, 3),
                    solver=rng.choice(["JACOBI", "SGS", "LINE"]), sweeps=rng.randint(4, 12), mixed=mixed, lag=1,
                    renumber=rng.choice([0, 1]), steps=rng.randint(4, 20), call=rng.choice(["march", "host"]))
    cells = _log_uniform(rng, 5.0e3, 7.0e5)
    ny = max(8, int(math.sqrt(cells / 4.0) * rng.uniform(0.8, 1.25)))
    nz = rng.randint(1, 3)
    return dict(kind="bump", nx=max(8, int(cells / (ny * nz))), ny=ny, nz=nz,
                flux=rng.choice(["HLLC", "HLLC", "HLLC", "ROE", "AUSM", "HAENEL"]), order2=rng.random() < 0.85,
                solver=rng.choice(["JACOBI", "SGS", "SGS"]), sweeps=rng.randint(4, 12), mixed=mixed,
                lag=rng.choice([1, SGS_LAG]), renumber=rng.choice([0, 1, 2]), steps=rng.randint(1, 10),
                call=rng.choice(["march", "host"]))


# ---------------------------------------------------------------------------
# meshes: the geometry of myjoe_b200.meshgen's channel bump and flat plate, extruded along z and
# formed with whole-array expressions (a 2M-cell mesh in seconds); boundary zones first
# ---------------------------------------------------------------------------
def _extruded(X, Y, z, zone_of):
    nx, ny, nz = X.shape[0] - 1, X.shape[1] - 1, len(z) - 1
    n2, dz, zm = nx * ny, np.diff(z), 0.5 * (z[1:] + z[:-1])
    P = np.stack([X, Y], -1)
    quad = np.stack([P[:-1, :-1], P[1:, :-1], P[1:, 1:], P[:-1, 1:]], 2)           # (i, j) cells, counter-clockwise
    nxt = np.roll(quad, -1, 2)
    cr = quad[..., 0] * nxt[..., 1] - nxt[..., 0] * quad[..., 1]
    area = 0.5 * cr.sum(2)
    cen = ((quad + nxt) * cr[..., None]).sum(2) / (6.0 * area[..., None])
    cid = np.arange(n2).reshape(ny, nx).T                                          # id within a layer
    lay = np.arange(nz)[:, None] * n2

    def side(a, b, c0, c1, sign):   # vertical faces over the 2-D edges a -> b, for every layer
        e = b - a
        n = np.stack([e[..., 1], -e[..., 0]], -1).reshape(-1, 2) * sign
        mid = (0.5 * (a + b)).reshape(-1, 2)
        fn = np.concatenate([n[None] * dz[:, None, None], np.zeros((nz, n.shape[0], 1))], -1).reshape(-1, 3)
        fx = np.concatenate([np.broadcast_to(mid, (nz,) + mid.shape),
                             np.broadcast_to(zm[:, None, None], (nz, mid.shape[0], 1))], -1).reshape(-1, 3)
        cv = np.stack([(lay + c0.ravel()).ravel(),
                       np.full(nz * c0.size, -1) if c1 is None else (lay + c1.ravel()).ravel()], 1)
        return cv, fx, fn

    def plane(k, sign):             # the z plane below layer k
        fx = np.concatenate([cen.transpose(1, 0, 2).reshape(-1, 2), np.full((n2, 1), z[k])], 1)
        fn = np.zeros((n2, 3))
        fn[:, 2] = sign * area.T.ravel()
        return fx, fn

    bnd = {}
    xa, xb, ya, yb = P[:, :-1], P[:, 1:], P[:-1, :], P[1:, :]
    parts = [("imin", side(xa[0], xb[0], cid[0], None, -1.0)), ("imax", side(xa[-1], xb[-1], cid[-1], None, 1.0)),
             ("jmin", side(ya[:, 0], yb[:, 0], cid[:, 0], None, 1.0)),
             ("jmax", side(ya[:, -1], yb[:, -1], cid[:, -1], None, -1.0))]
    for k, sign, c in ((0, -1.0, np.arange(n2)), (nz, 1.0, np.arange(n2) + (nz - 1) * n2)):
        parts.append(("kmin" if k == 0 else "kmax",
                      (np.stack([c, np.full(n2, -1)], 1),) + plane(k, sign)))
    for name, (cv, fx, fn) in parts:
        zn = np.array(zone_of(name, fx))
        for zname in dict.fromkeys(zn.tolist()):
            m = zn == zname
            bnd.setdefault(zname, []).append((cv[m], fx[m], fn[m]))
    zones, blocks, pos = [], [], 0
    for zname, lst in bnd.items():
        cnt = sum(len(b[0]) for b in lst)
        zones.append((zname, pos, pos + cnt - 1))
        blocks += lst
        pos += cnt
    blocks.append(side(xa[1:-1], xb[1:-1], cid[:-1], cid[1:], 1.0))
    blocks.append(side(ya[:, 1:-1], yb[:, 1:-1], cid[:, :-1], cid[:, 1:], -1.0))
    for k in range(1, nz):
        c = np.arange(n2) + (k - 1) * n2
        blocks.append((np.stack([c, c + n2], 1),) + plane(k, 1.0))
    cvofa = np.concatenate([b[0] for b in blocks]).astype(np.int32)
    x_fa = np.concatenate([b[1] for b in blocks])
    fa_n = np.concatenate([b[2] for b in blocks])
    ncv = n2 * nz
    x_cv = np.empty((nz, n2, 3))
    x_cv[..., :2] = cen.transpose(1, 0, 2).reshape(-1, 2)
    x_cv[..., 2] = zm[:, None]
    x_cv = x_cv.reshape(-1, 3)
    vol = (dz[:, None] * area.T.ravel()).ravel()
    # internal normals point from cvofa[f][0] to cvofa[f][1], boundary normals outward
    inn = np.arange(pos, len(cvofa))
    d = x_cv[cvofa[inn, 1]] - x_cv[cvofa[inn, 0]]
    fa_n[inn] *= np.sign((d * fa_n[inn]).sum(1))[:, None]
    out = np.arange(pos)
    fa_n[out] *= np.sign(((x_fa[out] - x_cv[cvofa[out, 0]]) * fa_n[out]).sum(1))[:, None]
    faocv_i, faocv_v = geometry.build_faocv(cvofa, ncv)
    nb_i, nb_v = geometry.build_nbocv(cvofa, ncv, pos)
    lsq, blsq = geometry.calc_lsg_coeff(x_cv, x_fa, cvofa, nb_i, nb_v, faocv_i, faocv_v, pos, ncv)
    return types.SimpleNamespace(ncv=ncv, nfa=len(cvofa), nfa_b=pos, cvofa=cvofa, faocv_i=faocv_i, faocv_v=faocv_v,
                                 nbocv_i=nb_i, nbocv_v=nb_v, x_cv=x_cv, x_fa=x_fa, fa_normal=fa_n, cv_volume=vol,
                                 nbocv_lsg_coeff=lsq, boundary_fa_lsg_coeff=blsq, zones=zones)


def _bump_mesh(nx, ny, nz, bump_h):
    xs = np.linspace(0.0, 3.0, nx + 1)
    yb = np.where((xs >= 1.0) & (xs <= 2.0), bump_h * np.sin(math.pi * (xs - 1.0)) ** 2, 0.0)
    Y = yb[:, None] + (1.0 - yb[:, None]) * np.linspace(0.0, 1.0, ny + 1)[None, :]
    names = {"imin": "inlet", "imax": "outlet", "jmin": "lower", "jmax": "upper", "kmin": "sides", "kmax": "sides"}
    return _extruded(np.repeat(xs[:, None], ny + 1, 1), Y, np.linspace(0.0, nz * 3.0 / nx, nz + 1),
                     lambda s, fx: [names[s]] * len(fx))


def _plate_mesh(nx, ny, nz, length, re_l):
    dy = 0.5 * length / (re_l * math.sqrt(0.664 / math.sqrt(re_l) / 2.0))
    xs = np.linspace(-0.25 * length, length, nx + 1)
    ys = np.concatenate([[0.0], np.cumsum(dy * 1.1 ** np.arange(ny))])
    names = {"imin": "inlet", "imax": "outlet", "jmax": "upper", "kmin": "sides", "kmax": "sides"}

    def zone(s, fx):
        return np.where(fx[:, 0] < 0.0, "lower_sym", "plate").tolist() if s == "jmin" else [names[s]] * len(fx)

    return _extruded(np.repeat(xs[:, None], ny + 1, 1), np.repeat(ys[None, :], nx + 1, 0),
                     np.linspace(0.0, nz * 1.25 * length / nx, nz + 1), zone)


@functools.lru_cache(maxsize=4)
def _mesh(kind, nx, ny, nz, n_prism=0, stretch=1.0, bump_h=0.1, mach=0.5, aoa=0.0):
    """The mesh and the flow settings: what a user's program reads from its mesh file and Joe.in."""
    if kind == "bump":
        prm = jcase.bump_case(8, 4, 1, mach=mach, inlet="FARFIELD", aoa_deg=aoa, bump_h=bump_h)[2]
        return _bump_mesh(nx, ny, nz, bump_h), prm
    if kind == "plate":
        prm = jcase.plate_case(8, 4, 1)[2]
        mu = prm.MU_REF * (prm.T_REF / prm.SL_TREF) ** 1.5 * (prm.SL_TREF + prm.SL_SREF) / (prm.T_REF + prm.SL_SREF)
        return _plate_mesh(nx, ny, nz, 1.0e5 * mu / (prm.RHO_INITIAL * prm.U_INITIAL[0]), 1.0e5), prm
    _, g, prm = jcase.sa_bump_case(nx, ny, nz, mach=0.7, re=3.0e6, bump_h=0.05, stretch=stretch, n_prism=n_prism,
                                   alternate=n_prism > 0, shuffle=True)
    return g, prm


@functools.lru_cache(maxsize=2)
def _batch_meshes(model, cases, lo, hi, pick):
    specs = [s for s in batch.case_specs(cases, lo, hi, pick)]
    out = []
    for s in specs:
        if model == "SST":
            out.append(batch.build_case(dict(s, model="SST", aoa=0.5 * s["aoa"])))
        else:
            out.append(_mesh("bump", s["nx"], s["ny"], s["nz"], bump_h=s["bump"], mach=min(s["mach"], 0.6),
                             aoa=s["aoa"]))
    return out


def _settings(case, prm):
    cfl = {"plate": 5.0, "sa": 20.0, "bump": 5.0}.get(case["kind"], 20.0 if case.get("model") == "SST" else 5.0)
    more = dict(SECOND_ORDER=case["order2"], SPACE_INTEGRATION=case["flux"]) if case["kind"] == "bump" else {}
    if case["kind"] == "sa":
        more = dict(SECOND_ORDER=False)
    return dataclasses.replace(prm, LINEAR_SOLVER_NS=case["solver"], LS_MAX_ITER=case["sweeps"], CFL=1.0,
                               CFL_RAMP=(10, 5, 1.2, cfl), **more)


def _state(x_cv, prm, rng):
    """The free stream times (1 + small smooth waves with phases and directions from the seed)."""
    lo, hi = x_cv.min(0), x_cv.max(0)
    s = (x_cv - lo) / np.maximum(hi - lo, 1e-300)

    def wave(a):
        k, ph = rng.uniform(1.0, 4.0, 3), rng.uniform(0.0, 2.0 * math.pi, 2)
        return a * np.sin(k[0] * s[:, 0] + k[2] * s[:, 2] + ph[0]) * np.cos(k[1] * s[:, 1] + ph[1])

    rho = prm.RHO_INITIAL * (1.0 + wave(0.01))
    u = np.asarray(prm.U_INITIAL, float)
    um = math.sqrt(float(u @ u))
    v = np.stack([u[0] + um * wave(0.02), u[1] + um * wave(0.01), u[2] + 0.0 * s[:, 0]], 1)
    p = prm.P_INITIAL * (1.0 + wave(0.01))
    return rho, rho[:, None] * v, p / (prm.GAMMA - 1.0) + 0.5 * rho * (v * v).sum(1)


def _scalars(g, prm, rng):
    f = 1.0 + 0.05 * np.sin(rng.uniform(1, 3) * g.x_cv[:, 0] + rng.uniform(0, 6)) * np.cos(
        rng.uniform(1, 3) * g.x_cv[:, 1])
    if prm.TURB_MODEL == "SA":
        return prm.NUSA_INITIAL * f
    return np.stack([prm.KINE_INITIAL * f, prm.OMEGA_INITIAL * np.ones(g.ncv)], 1)


def _flow(case):
    g, prm = _mesh(case["kind"], case["nx"], case["ny"], case["nz"], case.get("n_prism", 0),
                   case.get("stretch", 1.0))
    return g, _settings(case, prm)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    n = t.numpy()
    n[...] = a
    return n


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = types.SimpleNamespace(case=case)
    if case["kind"] == "batch":
        cs = [(g, _settings(case, p)) for g, p in
              _batch_meshes(case["model"], case["cases"], case["lo"], case["hi"], case["pick"])]
        s.b = solver.JoeGpuBatch(cs, precision=int(case["mixed"]), jac_lag=case["lag"], renumber=case["renumber"])
        for k, (g, p) in enumerate(cs):
            s.b.set_case_state(k, *_state(g.x_cv, p, rng))
            if p.TURB_MODEL != "NONE":
                s.b.set_case_scalars(k, _scalars(g, p, rng))
        return s
    g, prm = _flow(case)
    s.j = solver.JoeGpu(g, prm, precision=int(case["mixed"]), renumber=case["renumber"], jac_lag=case.get("lag", 1))
    s.q = _state(g.x_cv, prm, rng)
    if case["call"] == "host":
        s.q = tuple(_pinned(a) for a in s.q)
        s.resid = _pinned(np.zeros((case["steps"], 5)))
    else:
        s.j.set_state(*s.q)
        if case["kind"] == "sa":
            s.j.set_scalars(_scalars(g, prm, rng))
    return s


def run(s):
    case = s.case
    if case["kind"] == "batch":
        r = s.b.runBackwardEulerCases(case["steps"])
        out = [s.b.get_case_state(k) for k in range(s.b.ncases)]
        if case["model"] == "SST":
            phi = [s.b.get_case_scalars(k) for k in range(s.b.ncases)]
            return {"resid": r, "scalars": np.concatenate(phi), **_joined(out)}
        return {"resid": r, **_joined(out)}
    if case["call"] == "host":
        s.j.step_host(*s.q, case["steps"], s.resid)
        return {"resid": s.resid, "rho": s.q[0], "rhou": s.q[1], "rhoE": s.q[2]}
    if case["call"] == "restart":
        s.j.set_state(*s.q)
    r = s.j.runBackwardEuler(case["steps"])
    out = {"resid": r, **dict(zip(("rho", "rhou", "rhoE"), s.j.get_state()))}
    if case["kind"] == "sa":
        out["scalars"] = s.j.get_scalars()
    return out


def _joined(states):
    """The cases' states one after another (a batch of two dozen has too many arrays to name each)."""
    return {n: np.concatenate([q[i] for q in states]) for i, n in enumerate(("rho", "rhou", "rhoE"))}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: per step, the mesh (geometry, connectivity, least-squares coefficients) and the state read
    once, the new state written once, the implicit matrix written once and read once per sweep (it is an
    operand of every sweep and larger than the chip's registers), the sweeps' vectors.  Flops: about 2,000
    per internal face and step for reconstruction, flux and both 5 x 5 matrices (3,500 viscous, 6,000 with
    a turbulence model), the gradients, and the sweeps' block products."""
    B = {"sa": 6}.get(case["kind"], 7 if case.get("model") == "SST" else 5)
    if case["kind"] == "batch":
        cells = sum(2 * s["ny"] * s["ny"] * s["nz"] for s in
                    batch.case_specs(case["cases"], case["lo"], case["hi"], case["pick"]))
        nz = 2
    else:
        cells, nz = case["nx"] * case["ny"] * case["nz"], case["nz"]
        if case["kind"] == "sa":
            cells += case["nx"] * case["nz"] * case["n_prism"]   # each prism row holds two cells per quad
    f = 2.0 + (nz - 1.0) / nz                                    # internal faces per cell
    s = 4 if case["mixed"] else 8
    m = 1.0 + 2.0 * f
    turb = B > 5
    visc = turb or case["kind"] == "plate"
    geo = 8 * (3 + 1) + f * (8 * 6 + 4 * 4) + 8 * 3 * m
    state = 2 * 8 * B
    forms = 1.0 / case.get("lag", 1)
    matrix = s * B * B * m
    sweep = matrix + s * 3 * B + 4 * (m - 1)
    ls = 4 * case["sweeps"] // 2 if case["solver"] == "BCGSTAB" else case["sweeps"]
    per = geo + state + forms * matrix + ls * sweep
    flops = f * (6000 if turb else 3500 if visc else 2000) + m * 60 + ls * 2 * B * B * m
    return {"bytes": case["steps"] * cells * per, "flops": case["steps"] * cells * flops}


# ---------------------------------------------------------------------------
# the inviscid HLLC iteration in plain 64-bit torch
# ---------------------------------------------------------------------------
def _prims(q, gam):
    r = q[:, 0]
    u = q[:, 1:4] / r[:, None]
    p = (gam - 1.0) * (q[:, 4] - 0.5 * r * (u * u).sum(1))
    return torch.cat([r[:, None], u, p[:, None]], 1)


def _hllc(L, R, n, gam, waves=None):
    """HLLC flux per unit area of primitive states (rho, u, p); waves: fixed outer wave speeds."""
    def side(W):
        un = (W[:, 1:4] * n).sum(1)
        return W[:, 0], W[:, 1:4], W[:, 4], un, W[:, 4] / (gam - 1.0) + 0.5 * W[:, 0] * (W[:, 1:4] ** 2).sum(1)
    rl, ul, pl, unl, el = side(L)
    rr, ur, pr, unr, er = side(R)
    if waves is None:
        wl = 1.0 / (1.0 + torch.sqrt(rr / rl))
        wr = 1.0 - wl
        un = wl * unl + wr * unr
        u = wl[:, None] * ul + wr[:, None] * ur
        H = wl * (el + pl) / rl + wr * (er + pr) / rr
        c = torch.sqrt((gam - 1.0) * (H - 0.5 * (u * u).sum(1)))
        sl = torch.minimum(un - c, unl - torch.sqrt(gam * pl / rl))
        sr = torch.maximum(un + c, unr + torch.sqrt(gam * pr / rr))
    else:
        sl, sr = waves
    sm = (pl - pr - rl * unl * (sl - unl) + rr * unr * (sr - unr)) / (rr * (sr - unr) - rl * (sl - unl))
    ps = rr * (unr - sr) * (unr - sm) + pr

    def plain(r, u, p, un, e):
        return torch.cat([(r * un)[:, None], (r * un)[:, None] * u + p[:, None] * n, ((e + p) * un)[:, None]], 1)

    def star(r, u, p, un, e, s):
        f = (s - un) / (s - sm)
        ru = (r * f)[:, None] * u + ((ps - p) / (s - sm))[:, None] * n
        es = ((s - un) * e - p * un + ps * sm) / (s - sm)
        return torch.cat([(r * f * sm)[:, None], ru * sm[:, None] + ps[:, None] * n, ((es + ps) * sm)[:, None]], 1)

    left = torch.where((sl > 0.0)[:, None], plain(rl, ul, pl, unl, el), star(rl, ul, pl, unl, el, sl))
    right = torch.where((sr < 0.0)[:, None], plain(rr, ur, pr, unr, er), star(rr, ur, pr, unr, er, sr))
    return torch.where((sm >= 0.0)[:, None], left, right), (sl, sr)


def _hllc_matrices(QL, QR, n, gam):
    """d flux / d conserved states of both sides, the outer wave speeds held fixed."""
    waves = _hllc(_prims(QL, gam), _prims(QR, gam), n, gam)[1]
    AL, AR = [], []
    for k in range(5):
        e = torch.zeros_like(QL)
        e[:, k] = 1.0
        z = torch.zeros_like(QL)
        g = lambda a, b: _hllc(_prims(a, gam), _prims(b, gam), n, gam, waves)[0]  # noqa: E731
        AL.append(torch.func.jvp(g, (QL, QR), (e, z))[1])
        AR.append(torch.func.jvp(g, (QL, QR), (z, e))[1])
    return torch.stack(AL, 2), torch.stack(AR, 2)


def _bj(phi, grad, x_fa, x_cv, c0, c1, eps2, cut):
    """Limited gradients of one field: the smallest smooth ratio over a cell's internal faces."""
    hi, lo, ratio = phi.clone(), phi.clone(), torch.ones_like(phi)
    for a, b in ((c0, c1), (c1, c0)):
        hi.scatter_reduce_(0, a, phi[b], "amax")
        lo.scatter_reduce_(0, a, phi[b], "amin")
    for a in (c0, c1):
        dm = ((x_fa - x_cv[a]) * grad[a]).sum(1)
        dp = torch.where(dm >= 0.0, hi[a] - phi[a], lo[a] - phi[a])
        r = (dp * dp + 2.0 * dm * dp + eps2[a]) / (dp * dp + 2.0 * dm * dm + dm * dp + eps2[a])
        ratio.scatter_reduce_(0, a, r, "amin")
    return grad * torch.where(hi - lo > cut, ratio, torch.zeros_like(ratio))[:, None]


def _far_field(W, n, v, gam):
    """Riemann-invariant far field: the boundary state of the cell states W against the stream v."""
    u0, p0, r0 = v[:3], v[3], v[4]
    g1 = 2.0 / (gam - 1.0)
    cb = math.sqrt(gam * p0 / r0)
    qb, qe = (n * u0).sum(1), (n * W[:, 1:4]).sum(1)
    ce = torch.sqrt(gam * W[:, 4] / W[:, 0])
    a1 = torch.where(qb > -cb, qe + g1 * ce, qb + g1 * cb)
    a2 = torch.where(qb > cb, qe - g1 * ce, qb - g1 * cb)
    qn, cf = 0.5 * (a1 + a2), 0.25 * (a1 - a2) * (gam - 1.0)
    out = qb > 0.0
    u = torch.where(out[:, None], W[:, 1:4] + (qn - qe)[:, None] * n, u0 + (qn - qb)[:, None] * n)
    sf = torch.where(out, W[:, 0] ** gam / W[:, 4], torch.full_like(qb, float(r0 ** gam / p0)))
    r = (sf * cf * cf / gam) ** (1.0 / (gam - 1.0))
    return torch.cat([r[:, None], u, (r * cf * cf / gam)[:, None]], 1)


def exact(case, seed):
    if case["kind"] != "bump" or case["flux"] != "HLLC":
        return None
    cells = case["nx"] * case["ny"] * case["nz"]
    if cells * case["steps"] > 150_000 or (case["solver"] == "SGS" and case["renumber"] != 0):
        return None   # too long here, or relaxed colour by colour in an order of the handle's own
    g, prm = _flow(case)
    gam, T = prm.GAMMA, torch.from_numpy
    q0 = _state(g.x_cv, prm, np.random.default_rng(seed))
    Q = torch.cat([T(q0[0])[:, None], T(q0[1]), T(q0[2])[:, None]], 1)
    N, nb = g.ncv, g.nfa_b
    x_cv, x_fa, fn, vol = T(g.x_cv), T(g.x_fa), T(g.fa_normal), T(g.cv_volume)
    area = fn.norm(dim=1)
    n = fn / area[:, None]
    cv = T(g.cvofa.astype(np.int64))
    b0, c0, c1 = cv[:nb, 0], cv[nb:, 0], cv[nb:, 1]
    ni, ai, nbd, ab = n[nb:], area[nb:], n[:nb], area[:nb]
    lsq, blsq = T(g.nbocv_lsg_coeff), T(g.boundary_fa_lsg_coeff)
    row = T(np.repeat(np.arange(N), np.diff(g.nbocv_i)))
    col = T(g.nbocv_v.astype(np.int64))
    kind = [""] * nb
    for name, f0, f1 in g.zones:
        kind[f0:f1 + 1] = [prm.bcs[name].kind] * (f1 - f0 + 1)
    far, sym, wall = (torch.tensor([k == w for k in kind]) for w in ("FARFIELD", "SYMMETRY", "WALL"))
    vff = torch.tensor(prm.bcs["inlet"].values, dtype=torch.float64)
    hexcol = np.indices((case["nz"], case["ny"], case["nx"])).sum(0).ravel() % 2   # first-fit colours of a hex block
    rel = min(1.0, prm.UNDER_RELAXATION)
    cfl, step, resid, due, after = prm.CFL, 0, [], 0, prm.CFL_RAMP
    for _ in range(case["steps"]):
        step += 1
        if step >= after[0] and step % after[1] == 0 and cfl < after[3]:
            cfl *= after[2]
        W = _prims(Q, gam)
        c = torch.sqrt(gam * W[:, 4] / W[:, 0])
        Wb = W[b0].clone()
        un = (Wb[:, 1:4] * nbd).sum(1)
        Wb[:, 1:4] = torch.where(sym[:, None], Wb[:, 1:4] - un[:, None] * nbd, Wb[:, 1:4])
        Wb[:, 1:4] = torch.where(wall[:, None], torch.zeros(3, dtype=torch.float64), Wb[:, 1:4])
        Wb = torch.where(far[:, None], _far_field(W[b0], nbd, vff, gam), Wb)
        # the largest wave speed over a cell's faces
        lam = torch.zeros(N, dtype=torch.float64)
        for a, nn, ar in ((c0, ni, ai), (c1, ni, ai), (b0, nbd, ab)):
            lam.scatter_reduce_(0, a, ((W[a, 1:4] * nn).sum(1).abs() + c[a]) * ar, "amax")
        dt = cfl * vol / lam
        L, R, Lb = W[c0], W[c1], W[b0]
        if case["order2"]:
            grads = []
            for k in range(5):
                gk = torch.zeros(N, 3, dtype=torch.float64).index_add_(0, row, lsq * W[col, k][:, None])
                gk.index_add_(0, b0, blsq * Wb[:, k][:, None])
                ref = c if 1 <= k <= 3 else W[:, k].abs()
                e = prm.EPS * ref
                e = e if 1 <= k <= 3 else e.clamp(min=1e-8)
                if prm.LIMITER:
                    gk = _bj(W[:, k].contiguous(), gk, x_fa[nb:], x_cv, c0, c1, e * e, 1e-8 if 1 <= k <= 3 else 1e-12)
                grads.append(gk)
            G = torch.stack(grads, 1)

            def at(a, x):
                rec = W[a] + (G[a] * (x - x_cv[a])[:, None, :]).sum(2)
                ok = (rec[:, 0] > 0.0) & (rec[:, 4] > 0.0)
                return torch.where(ok[:, None], rec, W[a])

            L, R, Lb = at(c0, x_fa[nb:]), at(c1, x_fa[nb:]), at(b0, x_fa[:nb])
        F = _hllc(L, R, ni, gam)[0] * ai[:, None]
        solid = ~far
        Fb = torch.where(solid[:, None], _hllc(Wb, Wb, nbd, gam)[0], _hllc(Lb, Wb, nbd, gam)[0]) * ab[:, None]
        rhs = torch.zeros(N, 5, dtype=torch.float64).index_add_(0, c0, -F).index_add_(0, c1, F)
        rhs.index_add_(0, b0, -Fb)
        resid.append(rhs.abs().sum(0))
        if step >= due:
            due = step + case["lag"]
            AL, AR = (A * ai[:, None, None] for A in _hllc_matrices(Q[c0], Q[c1], ni, gam))
            Qb = torch.cat([Wb[:, :1], Wb[:, :1] * Wb[:, 1:4],
                            (Wb[:, 4] / (gam - 1.0) + 0.5 * Wb[:, 0] * (Wb[:, 1:4] ** 2).sum(1))[:, None]], 1)
            Ab = _hllc_matrices(torch.where(solid[:, None], Qb, Q[b0]), Qb, nbd, gam)[0] * ab[:, None, None]
            D0 = torch.zeros(N, 5, 5, dtype=torch.float64).index_add_(0, c0, AL).index_add_(0, c1, -AR)
            D0.index_add_(0, b0, Ab)
        Di = torch.linalg.inv(D0 + (vol / dt)[:, None, None] * torch.eye(5, dtype=torch.float64))
        b, x = rel * rhs, torch.zeros(N, 5, dtype=torch.float64)

        def relaxed():
            off = torch.zeros(N, 5, dtype=torch.float64)
            off.index_add_(0, c0, torch.bmm(AR, x[c1][:, :, None])[:, :, 0])
            off.index_add_(0, c1, -torch.bmm(AL, x[c0][:, :, None])[:, :, 0])
            return torch.bmm(Di, (b - off)[:, :, None])[:, :, 0]

        for it in range(case["sweeps"]):
            if case["solver"] == "JACOBI":
                x = relaxed()
            else:
                for k in ((0, 1) if it % 2 == 0 else (1, 0)):
                    x = torch.where(T(hexcol == k)[:, None], relaxed(), x)
        Q = Q + x
    return {"resid": torch.stack(resid).numpy(), "rho": Q[:, 0].contiguous().numpy(),
            "rhou": Q[:, 1:4].contiguous().numpy(), "rhoE": Q[:, 4].contiguous().numpy()}
