"""The work that a user of this framework has it do, as cases that can be timed and checked.

A case is one lattice (or a batch of them) and one pass over it, through the public entry
points of ``nonnewlbm_b200.Lattice``.  Three kinds of pass:

* ``frame``: upload the pulsating inflow rows of the next ``steps`` steps, take the steps, read
  the FP64 mass / flux sums and the macroscopic fields back (the loop of the studies: steps to
  the next output, then the output);
* ``coupled``: one step per call, each with its own inflow row, the sums of every step read back
  one step behind (a lattice coupled to a lumped circulation model), then the fields;
* ``driver``: the steps to the next output with mean/rms sums, then the 20 output fields of
  the result file (the loop of the TCPC driver).

The geometries are the repository's synthetic ones: a TCPC-like junction (5 % of its box is
fluid), a pipe, and a dense box that is periodic in y and z.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G
from nonnewlbm_b200 import units

FIELDS = (capi.M_RHO, capi.M_VX, capi.M_VY, capi.M_VZ)
BLOOD = units.Material("cy_blood", 1060.0, 0.00345 / 1060.0, 0.056, 3.313, 2.0, 0.3568, True)
NEWTONIAN = units.Material("newtonian_blood", 1060.0, 3.3e-6, 3.3e-6 * 1060.0, 1.0, 2.0, 1.0, False)


def _case(name, kind, nx=0, ny=0, nz=0, scale=0.0, n_cases=1, collision="CUM", dtype="f32", cy_mode="none", material="blood",
          bounce_back="fullway", stats=False, tune=False, mode="frame", steps=100, nu=0.01):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, scale=scale, n_cases=n_cases, collision=collision, dtype=dtype, cy_mode=cy_mode,
             material=material, bounce_back=bounce_back, stats=stats, tune=tune, mode=mode, steps=steps, nu=nu)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small pipe advanced one step per call by a coupled 0-d model: the smallest calls,
        # launch and readback latency count
        _case("coupled_pipe_f32", "pipe", 96, 32, 32, mode="coupled", steps=128, nu=1.0 / 30.0),
        # the pipe validation run in double precision, mean/rms sums on
        _case("pipe_f64", "pipe", 96, 32, 32, dtype="f64", stats=True, steps=400, nu=1.0 / 30.0),
        # the driver's loop on a coarse junction in double precision (parity runs), a
        # Carreau-Yasuda material of its table, all result fields written out
        _case("driver_junction_f64", "junction", scale=0.4, dtype="f64", cy_mode="local-neq", material="gx", stats=True, tune=True,
              mode="driver", steps=300),
        # the headline junction: cumulant, Carreau-Yasuda blood, FP64 mean/rms sums, tuned
        _case("junction_f32", "junction", scale=1.0, cy_mode="local-neq", stats=True, tune=True, steps=2000),
        # the storage-precision study: entropic collision, 16-bit storage
        _case("junction_kbc_f16", "junction", scale=0.75, collision="KBC_N4", dtype="f16", cy_mode="local-neq", steps=3000),
        # link-wise walls with the LES collision
        _case("junction_halfway_mrt", "junction", scale=0.6, collision="MRT_LES", bounce_back="halfway", steps=2000),
        # the finite-difference Carreau-Yasuda coupling of the multi-rank solver
        _case("junction_refd", "junction", scale=0.5, cy_mode="ref-fd", steps=1000),
        # a parameter study: junctions of several sizes and both rheologies in one launch group
        _case("batch_f32", "batch", scale=0.5, n_cases=8, cy_mode="local-neq", tune=True, steps=1000),
        # a dense box with mean/rms sums
        _case("box_f32_stats", "box", 192, 144, 120, stats=True, tune=True, steps=600, nu=0.05 / 3),
        # the largest: the throughput box in 16-bit storage
        _case("box_f16", "box", 384, 288, 240, dtype="f16", tune=True, steps=600, nu=0.05 / 3),
        # odd sizes, BGK, the other 16-bit type
        _case("box_bf16_bgk_odd", "box", 211, 163, 137, collision="BGK", dtype="bf16", tune=True, steps=1000, nu=0.05 / 3),
        # the entropic collision on a dense box
        _case("box_kbc_f32", "box", 176, 144, 112, collision="KBC_N4", steps=800, nu=0.05 / 3),
    ]


def draw(rng):
    """One more case of the same kinds and ranges."""
    kind = rng.choice(["pipe", "junction", "junction", "box", "box", "batch"])
    dtype = rng.choice(["f32", "f32", "f16", "bf16", "f64"])
    collision = rng.choice(["CUM", "CUM", "CUM", "BGK", "MRT_LES", "KBC_N1", "KBC_N2", "KBC_N3", "KBC_N4", "KBC_C1", "KBC_C2",
                            "KBC_C3", "KBC_C4"])
    stats, tune = rng.random() < 0.4, rng.random() < 0.6
    if kind == "pipe":
        d = rng.randint(14, 56)
        return _case("", kind, int(math.exp(rng.uniform(math.log(24), math.log(300)))), d, d, collision=collision, dtype=dtype,
                     bounce_back=rng.choice(["fullway", "halfway"]), stats=stats, tune=tune,
                     mode=rng.choice(["frame", "coupled"]), steps=rng.randint(60, 200), nu=rng.uniform(0.015, 0.05))
    if kind == "box":
        cells = math.exp(rng.uniform(math.log(1e5), math.log(1e7)))
        a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
        e = cells ** (1.0 / 3.0)
        nx, ny, nz = (max(16, int(round(v))) for v in (e * a, e * b, e / (a * b)))
        return _case("", kind, nx, ny, nz, collision=collision, dtype=dtype, stats=stats, tune=tune,
                     steps=rng.randint(100, 300), nu=rng.uniform(0.01, 0.04))
    if kind == "batch":
        return _case("", kind, scale=rng.uniform(0.25, 0.5), n_cases=rng.randint(2, 20), collision=collision,
                     dtype=rng.choice(["f32", "f16", "bf16"]), cy_mode=rng.choice(["none", "local-neq"]), tune=tune,
                     steps=rng.randint(100, 300), nu=rng.uniform(0.01, 0.03))
    cy_mode = rng.choice(["none", "local-neq", "local-neq", "ref-fd"])
    mode = "driver" if dtype == "f64" and rng.random() < 0.5 else "coupled" if rng.random() < 0.2 else "frame"
    return _case("", kind, scale=rng.uniform(0.25, 0.9), collision="CUM" if cy_mode == "ref-fd" else collision, dtype=dtype,
                 cy_mode=cy_mode, material=rng.choice(["blood", "gx"]),
                 bounce_back="fullway" if cy_mode == "ref-fd" else rng.choice(["fullway", "fullway", "halfway"]),
                 stats=stats or mode == "driver", tune=tune, mode=mode, steps=rng.randint(100, 400), nu=rng.uniform(0.01, 0.03))


# ---------------------------------------------------------------------------------------
# what the user's program has in hand
# ---------------------------------------------------------------------------------------
def _scales(case):
    """The geometry scale of each lattice: a batch spreads its cases over [1, 1.5] of its scale."""
    n = case["n_cases"]
    return [case["scale"] * (1.0 + 0.5 * k / max(1, n - 1)) for k in range(n)] if case["kind"] == "batch" else [case["scale"]]


@lru_cache(maxsize=16)
def _wall(scale):
    return G.study_to_geometry(G.junction(scale=scale))


@lru_cache(maxsize=4)
def _map(kind, nx, ny, nz):
    return G.pipe_map(nx, ny, nz, 0.375 * ny) if kind == "pipe" else G.dense_box_map(nx, ny, nz)


def _shape(case, k=0):
    if case["kind"] in ("pipe", "box"):
        return case["nx"], case["ny"], case["nz"]
    return _wall(_scales(case)[k]).shape[::-1]


def _material(case, k):
    if case["kind"] == "batch":
        return BLOOD if k % 2 else NEWTONIAN
    return BLOOD if case["material"] == "blood" else units.material_by_name(case["material"])


def _spec(case, k):
    cy, mode = (0.0, 0.0, 2.0, 1.0), "none"
    if case["cy_mode"] != "none":
        mat = _material(case, k)
        u = units.lattice_units(mat, 0.25e-3 / _scales(case)[k], case["nu"])
        cy = (u["nu0"], u["lambda"], u["a"], u["n"])
        mode = case["cy_mode"] if mat.carreau_yasuda else "none"
    return CaseSpec(_shape(case, k), collision=case["collision"], dtype=case["dtype"], cy_mode=mode, nu=case["nu"], cy=cy,
                    bounce_back=case["bounce_back"])


def _inputs(case, k, seed):
    """The seeded inputs of lattice k: the initial uniform state, the inflow rows of a pass (in
    units of the open areas) and the inlet profile of a pipe or a box."""
    rng = np.random.default_rng([seed, k])
    n = case["steps"]
    u0 = rng.uniform(-0.01, 0.01, 3)
    rho0 = rng.uniform(0.995, 1.005)
    phase, amp = rng.uniform(0, 2 * np.pi, 2), rng.uniform(0.05, 0.2, 2)
    peak = np.array([0.03, 0.02]) * rng.uniform(0.8, 1.3, 2)
    # one heart beat per pass
    t = 2 * np.pi * np.arange(n) / n
    rows = np.ones((n, 3))
    rows[:, 0] = peak[0] * (1.0 + amp[0] * np.sin(t + phase[0]))
    rows[:, 1] = peak[1] * (1.0 + amp[1] * np.sin(t + phase[1]))
    rows[:, 2] = 1.0 + amp[0] * np.sin(t + phase[0])
    prof = None
    if case["kind"] in ("pipe", "box"):
        m, p = _map(case["kind"], *_shape(case))
        z, y = np.nonzero(m[:, :, 0] == G.MAP_INFLOW_EQ)
        ph = rng.uniform(0, 2 * np.pi, 4)
        wy, wz = 2 * np.pi * y / m.shape[1], 2 * np.pi * z / m.shape[0]
        prof = p * (0.04 * (1.0 + 0.1 * np.sin(wy + ph[0]) * np.sin(wz + ph[1])))[:, None]
        prof[:, 1] = 0.004 * p[:, 0] * np.sin(wz + ph[2])
        prof[:, 2] = 0.004 * p[:, 0] * np.sin(wy + ph[3])
    return rho0, u0, rows, prof


def prepare(case, seed):
    n = case["n_cases"]
    lat = Lattice([_spec(case, k) for k in range(n)])
    rows, flags = [], None
    for k in range(n):
        rho0, u0, r, prof = _inputs(case, k, seed)
        if case["kind"] in ("pipe", "box"):
            lat.set_map(_map(case["kind"], *_shape(case))[0], ic=k)
            lat.set_inflow_profile(prof, ic=k)
        else:
            wall = _wall(_scales(case)[k])
            a = lat.setup_tcpc(wall, ic=k)
            r = r * np.array([a["left_area"], a["right_area"], 1.0])
            lat.set_inflow(ivc_flux=r[0, 0], svc_flux=r[0, 1], ic=k)
            if case["mode"] == "driver":
                flags = capi.tcpc_labels(wall, with_wall_flags=True)[3]
        lat.init_equilibrium(rho0, *u0, ic=k)
        rows.append(r)
    if case["tune"]:
        lat.autotune(stats=case["stats"], macro=case["mode"] == "driver")
    return {"case": case, "lat": lat, "rows": rows, "flags": flags, "summed": 0}


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
# a single-precision run's results are kept in single precision, a 16-bit run's fields in half
# precision (the digits that its populations hold)
FIELD_TYPE = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16, "bf16": torch.float16}


def _sums_type(case):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _fields(lat, case, k):
    """Density and velocity of lattice k, [4][z][y][x]."""
    out = torch.empty((4,) + lat.shape(k), dtype=FIELD_TYPE[case["dtype"]])
    for j, f in enumerate(FIELDS):
        out[j] = torch.from_numpy(lat.macro(f, ic=k))
    return out


def _output_call(case, dx, dt, mat, conv):
    cy = (conv["nu0"], conv["lambda"], conv["a"], conv["n"]) if mat.carreau_yasuda else None
    return dict(dx=dx, dt=dt, density=mat.density, nu_lbm=dt / dx / dx * mat.nu_inf, cy=cy)


def _driver_units(case):
    mat = _material(case, 0)
    dx = 0.25e-3 / case["scale"]
    conv = units.lattice_units(mat, dx, case["nu"])
    return _output_call(case, dx, conv["dt"], mat, conv)


def run(state):
    case, lat, rows = state["case"], state["lat"], state["rows"]
    n, stats = case["steps"], case["stats"]
    if case["mode"] == "coupled":
        sums = np.empty((n, 5))
        for k in range(n):
            lat.set_schedule(rows[0][k:k + 1])
            lat.step(1, stats=stats, macro=k == n - 1, reduce=True, wait=False, readback=True)
            if k:
                sums[k - 1] = lat.readback()[0]
        sums[n - 1] = lat.readback()[0]
        return {"sums": sums.astype(_sums_type(case)), "fields": _fields(lat, case, 0)}
    for k in range(case["n_cases"]):
        lat.set_schedule(rows[k], ic=k)
    if case["mode"] == "driver":
        lat.step(n, stats=True, macro=True)
        state["summed"] += n
        return dict(lat.output_fields(steps_summed=state["summed"], wall_flags=state["flags"], **_driver_units(case)))
    lat.step(n, stats=stats, macro=True, reduce=True)
    sums = np.stack([lat.reduce(k) for k in range(case["n_cases"])]).astype(_sums_type(case))
    return {"sums": sums, "fields": [_fields(lat, case, k) for k in range(case["n_cases"])]}


def _cells(case):
    """(colliding cells, cells of the box) over the lattices of a case."""
    fluid = box = 0
    for k in range(case["n_cases"]):
        if case["kind"] in ("pipe", "box"):
            m = _map(case["kind"], *_shape(case))[0]
        else:
            m = capi.tcpc_labels(_wall(_scales(case)[k]))[0]
        fluid += int(((m == G.MAP_FLUID) | (m == G.MAP_PERIODIC)).sum())
        box += m.size
    return fluid, box


def work(case):
    fluid, box = _cells(case)
    s = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}[case["dtype"]]
    ct = 8 if case["dtype"] == "f64" else 4
    # every step reads and writes each colliding cell's 27 populations once, and its six
    # FP64 sums where they are kept; the results are written out once
    per_step = fluid * (54 * s + (96 if case["stats"] else 0))
    out = box * 80 if case["mode"] == "driver" else box * 4 * min(ct, FIELD_TYPE[case["dtype"]].itemsize)
    # about 27 x 3 moment sums and 27 x 8 operations to rebuild the populations
    return {"bytes": float(per_step * case["steps"] + out), "flops": float(fluid * 300 * case["steps"])}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch: the pull scheme on the cells that hold fluid, open-plane
# nodes and the walls next to them
# ---------------------------------------------------------------------------------------
C = [(q // 9 - 1, (q // 3) % 3 - 1, q % 3 - 1) for q in range(27)]


def _axis(u):
    return (3 * u * u - 3 * u + 1, 3 * u * u - 2, 3 * u * u + 3 * u + 1)


def _node_equilibrium(rho, u):
    """The factorised equilibrium as the solver ships it (its pmm population carries rho twice)."""
    X, Y, Z = (_axis(v) for v in u)
    pre = {0: -1 / 27, 1: 1 / 54, 2: -1 / 108, 3: 1 / 216}
    f = torch.stack([pre[sum(map(abs, c))] * rho * X[c[0] + 1] * Y[c[1] + 1] * Z[c[2] + 1] for c in C])
    f[18] = f[18] * rho
    return f


def _product_equilibrium(rho, u):
    def ax(v):
        z = v * v - 2 / 3
        p = -0.5 * (z + 1 + v)
        return (p + v, z, p)

    X, Y, Z = (ax(v) for v in u)
    return torch.stack([-rho * X[c[0] + 1] * Y[c[1] + 1] * Z[c[2] + 1] for c in C])


def _moment_matrix(dev):
    """Rows: 200 020 002 110 101 011 210 201 120 021 102 012 111 and 1, 100, 010, 001."""
    rows = [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1), (2, 1, 0), (2, 0, 1), (1, 2, 0), (0, 2, 1), (1, 0, 2),
            (0, 1, 2), (1, 1, 1), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    return torch.tensor([[c[0] ** a * c[1] ** b * c[2] ** d for c in C] for a, b, d in rows], dtype=torch.float64, device=dev)


def _shear_matrix(use_t, use_q, dev):
    """s_q from (T Nxz Nyz Pxy Pxz Pyz Qxxy Qxxz Qxyy Qyyz Qxzz Qyzz Qxyz)."""
    S = torch.zeros(27, 13, dtype=torch.float64)
    for q, (x, y, z) in enumerate(C):
        k = abs(x) + abs(y) + abs(z)
        T = Q = None
        if k == 0:
            T = -1.0
        elif k == 1:
            S[q, 1], S[q, 2] = (2 / 6, -1 / 6) if x else (-1 / 6, 2 / 6) if y else (-1 / 6, -1 / 6)
            T = 1 / 6
            Q = {8: -x / 2, 10: -x / 2} if x else {6: -y / 2, 11: -y / 2} if y else {7: -z / 2, 9: -z / 2}
        elif k == 2:
            if not z:
                S[q, 3], Q = x * y / 4, {8: x / 4, 6: y / 4}
            elif not y:
                S[q, 4], Q = x * z / 4, {10: x / 4, 7: z / 4}
            else:
                S[q, 5], Q = y * z / 4, {11: y / 4, 9: z / 4}
        else:
            Q = {12: x * y * z / 8}
        if use_t and T is not None:
            S[q, 0] = T
        if use_q and Q:
            for j, v in Q.items():
                S[q, j] = v
    return S.to(dev)


def _viscosity(Cm, rho, p):
    """The local Carreau-Yasuda viscosity from the central second moments (xx yy zz xy xz yz) and
    the strain rate; p: nu_inf, nu0, lambda, a, n."""
    ninf, n0, lam, a, n = p
    P = [Cm[j] - rho / 3 for j in range(3)] + [Cm[j] for j in range(3, 6)]
    pn = torch.sqrt(P[0] ** 2 + P[1] ** 2 + P[2] ** 2 + 2 * (P[3] ** 2 + P[4] ** 2 + P[5] ** 2))
    K = 3 * math.sqrt(2.0) * pn / (2 * rho)
    t0 = torch.full_like(K, 3 * n0 + 0.5)
    t = t0
    for _ in range(3):
        s = (lam * K / t) ** a
        pw = (1 + s) ** ((n - 1) / a)
        g = t - 3 * (ninf + (n0 - ninf) * pw) - 0.5
        t = t - g / (1 + 3 * ((n0 - ninf) * (n - 1) * s * pw / (1 + s)) / t)
    t = torch.where(K > 0, t, t0)
    return (t - 0.5) / 3, [-3 / (2 * rho * t) * v for v in P]


def _cumulant(f, rho, u, om):
    k = f.reshape(3, 3, 3, -1)
    for ax, v in ((2, u[2]), (1, u[1]), (0, u[0])):
        m, z, p = k.unbind(ax)
        s, d = p + m, p - m
        k0 = s + z
        k = torch.stack([k0, d - v * k0, s - 2 * v * d + v * v * k0], ax)
    r = 1 / rho
    s = torch.zeros_like(k)
    k0 = k[0, 0, 0]
    a, b, c = (1 - om) * k[1, 1, 0], (1 - om) * k[1, 0, 1], (1 - om) * k[0, 1, 1]
    e1, e2 = (1 - om) * (k[2, 0, 0] - k[0, 2, 0]), (1 - om) * (k[2, 0, 0] - k[0, 0, 2])
    X, Y, Z = (e1 + e2 + k0) / 3, (e2 - 2 * e1 + k0) / 3, (e1 - 2 * e2 + k0) / 3
    s[0, 0, 0], s[1, 0, 0], s[0, 1, 0], s[0, 0, 1] = k0, -k[1, 0, 0], -k[0, 1, 0], -k[0, 0, 1]
    s[1, 1, 0], s[1, 0, 1], s[0, 1, 1], s[2, 0, 0], s[0, 2, 0], s[0, 0, 2] = a, b, c, X, Y, Z
    s[2, 1, 1], s[1, 2, 1], s[1, 1, 2] = (X * c + 2 * a * b) * r, (Y * b + 2 * a * c) * r, (Z * a + 2 * b * c) * r
    s[2, 2, 0], s[2, 0, 2], s[0, 2, 2] = (X * Y + 2 * a * a) * r, (X * Z + 2 * b * b) * r, (Y * Z + 2 * c * c) * r
    s[2, 2, 2] = (X * s[0, 2, 2] + Y * s[2, 0, 2] + Z * s[2, 2, 0] + 4 * (c * s[2, 1, 1] + b * s[1, 2, 1] + a * s[1, 1, 2])) * r - (
        16 * a * b * c + 4 * (b * b * Y + c * c * X + a * a * Z) + 2 * X * Y * Z) * r * r
    for ax, v in ((0, u[0]), (1, u[1]), (2, u[2])):
        k0, k1, k2 = s.unbind(ax)
        s = torch.stack([(k0 * (v * v - v) + k1 * (2 * v - 1) + k2) / 2, k0 * (1 - v * v) - 2 * v * k1 - k2,
                         (k0 * (v * v + v) + k1 * (2 * v + 1) + k2) / 2], ax)
    return s.reshape(27, -1)


def _les(f, rho, u, nu, M):
    P = list(M[:6] @ f)
    x, y, z = u
    N = [P[0] - rho * (1 / 3 + x * x), P[1] - rho * (1 / 3 + y * y), P[2] - rho * (1 / 3 + z * z), P[3] - rho * x * y, P[4] - rho * x * z,
         P[5] - rho * y * z]
    Q = 2 * (N[0] ** 2 + N[1] ** 2 + N[2] ** 2 + 2 * (N[3] ** 2 + N[4] ** 2 + N[5] ** 2))
    tau = 3 * nu + 0.5
    om = 2 / (torch.sqrt(tau * tau + 2 * 0.0342 * 9 * torch.sqrt(Q) / rho) + tau)
    P = [p - om * v for p, v in zip(P, N)]
    tr = P[0] + P[1] + P[2]
    out = []
    for cx, cy, cz in C:
        c2 = cx * cx + cy * cy + cz * cz
        pp = cx * cx * P[0] + cy * cy * P[1] + cz * cz * P[2] + 2 * (cx * cy * P[3] + cx * cz * P[4] + cy * cz * P[5])
        w = (8 / 27, 2 / 27, 1 / 54, 1 / 216)[c2]
        out.append(w * (rho * (2.5 - 1.5 * c2 + 3 * (cx * x + cy * y + cz * z)) + 4.5 * pp - 1.5 * tr))
    return torch.stack(out)


def _entropic(f, rho, u, nu, M, kind):
    central, v = kind[4] == "C", int(kind[5])
    x, y, z = u
    R = list(M[:13] @ f)
    T, Nxz, Nyz = R[0] + R[1] + R[2], R[0] - R[2], R[1] - R[2]
    if not central:
        xx, yy, zz = x * x, y * y, z * z
        m = [T, Nxz, Nyz, R[3], R[4], R[5], R[6], R[7], R[8], R[9], R[10], R[11], R[12]]
        e = [rho * (1 + xx + yy + zz), rho * (xx - zz), rho * (yy - zz), rho * x * y, rho * x * z, rho * y * z, rho * y * (1 / 3 + xx),
             rho * z * (1 / 3 + xx), rho * x * (1 / 3 + yy), rho * z * (1 / 3 + yy), rho * x * (1 / 3 + zz), rho * y * (1 / 3 + zz),
             rho * x * y * z]
    else:
        cT = T - rho * (x * x + y * y + z * z)
        a, b = Nxz + rho * (z * z - x * x), Nyz + rho * (z * z - y * y)
        pxy, pxz, pyz = R[3] - rho * x * y, R[4] - rho * x * z, R[5] - rho * y * z
        m = [cT, a, b, pxy, pxz, pyz, R[6] - (6 * x * pxy + y * (3 * x * x + 2 * a - b + cT)) / 3,
             R[7] - (6 * x * pxz + z * (3 * x * x + 2 * a - b + cT)) / 3, R[8] - (6 * y * pxy + x * (3 * y * y + 2 * b - a + cT)) / 3,
             R[9] - (6 * y * pyz + z * (3 * y * y + 2 * b - a + cT)) / 3, R[10] - (6 * z * pxz + x * (3 * z * z - b - a + cT)) / 3,
             R[11] - (6 * z * pyz + y * (3 * z * z - b - a + cT)) / 3, R[12] - x * pyz - y * pxz - z * pxy - x * y * z]
        e = [rho] + [torch.zeros_like(rho)] * 12
    ds = _shear_matrix(v in (2, 4), v in (3, 4), f.device) @ torch.stack([p - q for p, q in zip(m, e)])
    feq = _product_equilibrium(rho, u)
    dh = f - feq - ds
    num, den = (ds * dh / feq).sum(0), (dh * dh / feq).sum(0)
    beta = 1 / (6 * nu + 1)
    gamma = torch.where(den != 0, 1 / beta - (2 - 1 / beta) * num / den, 1 / beta + 0 * den)
    return f - beta * (2 * ds + gamma * dh)


def _exact_one(case, k, seed, dev):
    """(sums of every step [n][5], density and velocity [4][z][y][x], strain [6], mean/rms sums [6])."""
    spec = _spec(case, k)
    nx, ny, nz = spec.shape
    N = nx * ny * nz
    rho0, u0, rows, prof = _inputs(case, k, seed)
    lab = _map(case["kind"], nx, ny, nz)[0] if case["kind"] in ("pipe", "box") else capi.tcpc_labels(_wall(_scales(case)[k]))[0]
    L = torch.from_numpy(lab.astype(np.int64)).to(dev)
    half = spec.bounce_back == "halfway"
    D = dict(dtype=torch.float64, device=dev)
    # the cells that matter: all but walls with only walls around them
    live = (L != 1).to(torch.float32)[None, None]
    live = torch.nn.functional.max_pool3d(torch.nn.functional.pad(live, (1,) * 6, mode="circular"), 3, 1)[0, 0] > 0
    cells = torch.nonzero(live.reshape(-1)).reshape(-1)
    at = torch.zeros(N, dtype=torch.int64, device=dev)
    at[cells] = torch.arange(cells.numel(), device=dev)
    x, y, z = cells % nx, (cells // nx) % ny, cells // (nx * ny)
    lab = L.reshape(-1)[cells]

    def where(X, Y, Z):
        return at[X + nx * (Y + ny * Z)]

    def neighbours(x, y, z):
        return torch.stack([where((x - cx) % nx, (y - cy) % ny, (z - cz) % nz) for cx, cy, cz in C])

    def back(src):  # where a population comes from a wall, link-wise: the cell's own opposite one
        return (lab[src] == 1) if half else None

    src = neighbours(x, y, z)
    wall, moving = lab == 1, (lab == 0) | (lab == 2)
    fluid = torch.nonzero(moving).reshape(-1)
    wall_i = torch.nonzero(wall).reshape(-1)
    nodes = []  # (label, node, its inward cell, the stencil of that cell clamped around the node)
    for lb, (dx, dy) in {3: (1, 0), 4: (-1, 0), 5: (0, 1), 6: (0, -1), 8: (-1, 0)}.items():
        i = torch.nonzero(lab == lb).reshape(-1)
        if i.numel():
            X, Y, Z = x[i], y[i], z[i]
            st = []
            for cx, cy, cz in C:
                sx = (X + dx - cx) if dx else (X - cx)
                sy = (Y + dy - cy) if dy else (Y - cy)
                st.append(where(sx.clamp(0, nx - 1), sy.clamp(0, ny - 1), (Z - cz).clamp(0, nz - 1)))
            nodes.append((lb, i, where(X + dx, Y + dy, Z), torch.stack(st)))
    ineq = torch.nonzero(lab == 7).reshape(-1)
    P = torch.from_numpy(prof).to(dev) if prof is not None else None
    one = torch.ones(cells.numel(), **D)
    df = _node_equilibrium(rho0 * one, [v * one for v in u0])
    M = _moment_matrix(dev)
    flip = torch.arange(26, -1, -1, device=dev)
    nu, (n0, lam, a, n) = spec.nu, spec.cy
    sel = src[:, fluid]
    sel_back = back(sel)
    refd = spec.cy_mode == "ref-fd"
    if refd:
        fl = lab == 0
        near = [where((x + s * (j == 0)) % nx, (y + s * (j == 1)) % ny, (z + s * (j == 2)) % nz)[fluid] for j in range(3) for s in (-1, 1)]
        isf = [fl[i] for i in near]
    F = [torch.zeros(fluid.numel(), **D) for _ in range(3)]
    R, U = one.clone(), [torch.zeros_like(one) for _ in range(3)]
    strain = torch.zeros(6, cells.numel(), **D)
    stats = torch.zeros(6, cells.numel(), **D)
    sums = torch.zeros(rows.shape[0], 5, **D)

    def pull(idx, bk, own):
        f = torch.gather(df, 1, idx)
        return torch.where(bk, df[:, own][flip], f) if bk is not None else f

    def density_velocity(f, F):
        r, jx, jy, jz = M[13:17] @ f
        return r, [(j + 0.5 * g) / r for j, g in zip((jx, jy, jz), F)]

    def slope(v, axis):
        m, p, c = v[near[2 * axis]], v[near[2 * axis + 1]], v[fluid]
        fm, fp = isf[2 * axis], isf[2 * axis + 1]
        return torch.where(fm & fp, 0.5 * (p - m), torch.where(fm, c - m, torch.where(fp, p - c, torch.zeros_like(c))))

    zero3 = (0.0, 0.0, 0.0)
    for t in range(rows.shape[0]):
        f = pull(sel, sel_back, fluid)
        if refd:
            _, v = density_velocity(f, F)
            V = [torch.zeros_like(one) for _ in range(3)]
            for j in range(3):
                V[j][fluid] = v[j]
            s11, s22, s33 = slope(V[0], 0), slope(V[1], 1), slope(V[2], 2)
            s12, s13, s32 = ((slope(V[p], i) + slope(V[i], p)) / 2 for i, p in ((0, 1), (0, 2), (1, 2)))
            T = {}
            for key, s in (("11", s11), ("12", s12), ("13", s13), ("22", s22), ("32", s32), ("33", s33)):
                T[key] = torch.zeros_like(one)
                T[key][fluid] = s
            g = math.sqrt(2.0) * torch.sqrt(s11 ** 2 + s22 ** 2 + s33 ** 2 + 2 * (s12 ** 2 + s13 ** 2 + s32 ** 2))
            w = 2 * ((nu + (n0 - nu) * (1 + (g * lam) ** a) ** ((n - 1) / a)) - nu)
            F = [w * (slope(T[p], 0) + slope(T[q], 1) + slope(T[r], 2)) for p, q, r in (("11", "12", "13"), ("12", "22", "32"), ("13", "32", "33"))]
        rho, u = density_velocity(f, F)
        nuc = nu
        if spec.cy_mode == "local-neq":
            m = M @ f
            ux, uy, uz = u
            Cm = [m[0] - 2 * ux * m[14] + rho * ux * ux, m[1] - 2 * uy * m[15] + rho * uy * uy, m[2] - 2 * uz * m[16] + rho * uz * uz,
                  m[3] - ux * m[15] - uy * m[14] + rho * ux * uy, m[4] - ux * m[16] - uz * m[14] + rho * ux * uz,
                  m[5] - uy * m[16] - uz * m[15] + rho * uy * uz]
            nuc, S = _viscosity(Cm, rho, (nu, n0, lam, a, n))
            strain[:, fluid] = torch.stack(S)
        om = 1 / (3 * nuc + 0.5)
        if spec.collision == "CUM":
            post = _cumulant(f, rho, u, om)
        elif spec.collision == "BGK":
            post = f + (_product_equilibrium(rho, u) - f) * om
        elif spec.collision == "MRT_LES":
            post = _les(f, rho, u, nuc, M)
        else:
            post = _entropic(f, rho, u, nuc, M, spec.collision)
        new = torch.zeros_like(df)
        new[:, wall_i] = torch.gather(df, 1, src[:, wall_i])[flip]
        new[:, fluid] = post
        R[fluid] = rho
        for j in range(3):
            U[j][fluid] = u[j]
        ul, ur, ps = rows[t, 0], -rows[t, 1], rows[t, 2]
        for lb, i, inward, st in nodes:
            g = pull(st, back(st), inward)
            r, v = density_velocity(g, zero3)
            if lb in (3, 4):
                v = [torch.full_like(r, ul if lb == 3 else ur), torch.zeros_like(r), torch.zeros_like(r)]
            else:
                r = torch.ones_like(r)
            new[:, i] = _node_equilibrium(r, v)
            R[i] = r
            for j in range(3):
                U[j][i] = v[j]
            if lb != 8:
                sums[t, lb - 2] = {3: v[0], 4: -v[0], 5: -v[1], 6: v[1]}[lb].sum()
        if ineq.numel():
            r, v = torch.ones(ineq.numel(), **D), [P[:, j] * ps for j in range(3)]
            new[:, ineq] = _node_equilibrium(r, v)
            R[ineq] = r
            for j in range(3):
                U[j][ineq] = v[j]
        sums[t, 0] = rho.sum()
        if case["stats"]:
            for j in range(3):
                stats[j] += torch.where(wall, 0 * one, R * U[j])
                stats[3 + j] += torch.where(wall, 0 * one, (R * U[j]) ** 2)
        df = new
    out = torch.zeros(4, N, **D)
    out[0] = 1.0
    out[0, cells] = torch.where(wall, one, R)
    for j in range(3):
        out[1 + j, cells] = torch.where(wall, 0 * one, U[j])

    def full(v):
        o = torch.zeros(v.shape[0], N, **D)
        o[:, cells] = v
        return o.reshape(-1, nz, ny, nx)

    return sums, out.reshape(4, nz, ny, nx), full(strain), full(stats)


def _output_exact(case, fields, strain, stats, flags):
    d = _driver_units(case)
    dx, dt, dens, nul, cy = d["dx"], d["dt"], d["density"], d["nu_lbm"], d["cy"]
    v2p, n = dx / dt, case["steps"]
    vel = fields[1:] * v2p
    mean = stats[:3] * v2p / n
    r = (stats[3:] * v2p * v2p / n - mean * mean).abs()
    rms, mv = r.square().sum(0).sqrt(), mean.square().sum(0).sqrt()
    turb = torch.where(mv <= 1e-10, torch.zeros_like(mv), rms / mv.clamp(min=1e-300))
    xx, yy, zz, xy, xz, yz = strain
    gl = math.sqrt(2.0) * torch.sqrt(xx ** 2 + yy ** 2 + zz ** 2 + 2 * (xy ** 2 + xz ** 2 + yz ** 2))
    nu = nul + (cy[0] - nul) * (1 + (gl * cy[1]) ** cy[2]) ** ((cy[3] - 1) / cy[2]) if cy else torch.full_like(gl, nul)
    nup = nu * dx * dx / dt
    w = torch.from_numpy(flags.astype(np.float32)).to(fields.device).reshape(gl.shape)
    near = torch.zeros_like(w)
    near[1:] += w[:-1]
    near[:-1] += w[1:]
    near[:, 1:] += w[:, :-1]
    near[:, :-1] += w[:, 1:]
    near[:, :, 1:] += w[:, :, :-1]
    near[:, :, :-1] += w[:, :, 1:]
    wss = torch.where(near > 0, nup * dens * gl / dt, torch.zeros_like(gl))
    got = [vel, mean, fields[0], (fields[0] - 1) * dens * v2p * v2p / 3, gl / dt, nup, nup * dens, wss, turb, rms,
           torch.stack([xx, yy, zz]) / dt, torch.stack([xy, xz, yz]) / dt]
    return {name: v for (name, _), v in zip(capi.OUTPUT_FIELDS, got)}


def exact(case, seed):
    fluid, _ = _cells(case)
    # about 6 ms a step of a small lattice, 4 ns a cell and step of a large one
    if fluid * case["steps"] > 3e9 or case["n_cases"] * case["steps"] > 3000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["mode"] == "driver":
        _, fields, strain, stats = _exact_one(case, 0, seed, dev)
        return _output_exact(case, fields, strain, stats, capi.tcpc_labels(_wall(case["scale"]), with_wall_flags=True)[3])
    got = [_exact_one(case, k, seed, dev) for k in range(case["n_cases"])]
    if case["mode"] == "coupled":
        return {"sums": got[0][0], "fields": got[0][1]}
    return {"sums": torch.stack([g[0][-1] for g in got]), "fields": [g[1] for g in got]}
