"""The work that users of this framework have it do, as measurable cases.

One case is one call sequence through the public entry points: a solve of one
RVE (thermal, elastic, J2 or damage) with its field copied back, an effective
tensor of one or many RVEs, a plane solve, a reconstruction.  ``listed()``
names the cases that are always measured, ``draw(rng)`` gives further ones of
the same ranges, ``prepare`` makes what a user's program holds before the call
(the phase maps, the solver handle with its material and load, page-locked
memory for the results), ``run`` is one pass, ``work`` the bytes and operations
it cannot do without, and ``exact`` the results from plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import mat3d_b200 as m3d

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
# The line lengths of the published workloads, and what users bring besides.
COMMON = (32, 48, 64, 96, 128)


def listed():
    return [
        # a conduction solve of a small RVE: a sweep is a few microseconds of work, so latency and launches count
        {"name": "thermal_32", "kind": "thermal", "n": 32, "precision": "fp64", "rule": "residual", "tol": 1e-8, "contrast": 10.0},
        # the reference's own example grid length (65 = 5 x 13) under the reference's stop rule, as a ported driver runs it
        {"name": "thermal_65_ref", "kind": "thermal", "n": 65, "precision": "fp64", "rule": "reference", "tol": 1e-6, "contrast": 0.05},
        # the headline workload's grid, material and precision: 128^3 conduction at contrast 100, FP32 sweeps + FP64 refinement
        {"name": "thermal_128", "kind": "thermal", "n": 128, "precision": "fp32_refine", "rule": "residual", "tol": 1e-10, "contrast": 100.0},
        # the largest grid one RVE is solved on
        {"name": "thermal_256", "kind": "thermal", "n": 256, "precision": "fp32_refine", "rule": "residual", "tol": 1e-10, "contrast": 30.0},
        # the elastic validation workload: 64^3 spheres, FP64 to residual 1e-6
        {"name": "elastic_64", "kind": "elastic", "n": 64, "precision": "fp64", "rule": "residual", "tol": 1e-6, "contrast": 23.0},
        # batched homogenization, many small RVEs of mixed contrast with six load cases each
        {"name": "homog_32x24", "kind": "homog", "n": 32, "precision": "fp32_refine", "tol": 1e-9, "rves": 24},
        # batched homogenization at the grid size that carries most of the batch workload's voxels
        {"name": "homog_96x4", "kind": "homog", "n": 96, "precision": "fp32_refine", "tol": 1e-9, "rves": 4},
        # one RVE's effective stiffness on a grid length without a compile-time transform (75 = 3 x 5 x 5)
        {"name": "homog_75x1", "kind": "homog", "n": 75, "precision": "fp32_refine", "tol": 1e-9, "rves": 1},
        # elasto-plastic load steps under mixed control, FP32 transforms as the published J2 workload runs them
        {"name": "j2_64", "kind": "j2", "n": 64, "precision": "fp32", "tol": 1e-4, "increments": 3, "strain": 3e-3},
        # one load step past yield on the published workload's grid, FP64
        {"name": "j2_256", "kind": "j2", "n": 256, "precision": "fp64", "tol": 1e-4, "increments": 1, "strain": 1.5e-3},
        # plane homogenization: three load cases of 25 iterations
        {"name": "plane_1024", "kind": "plane", "n": 1024, "iterations": 25},
        # reconstruction passes on the reference example's 171^3 grid (171 = 9 x 19)
        {"name": "rec_171", "kind": "rec", "n": 171, "passes": 10},
    ]


def _length(rng, lo, hi, common=COMMON):
    """A grid length in [lo, hi], log-uniform (or a common one), whose prime factors the transforms take (<= 31)."""
    pool = [n for n in common if lo <= n <= hi]
    if pool and rng.random() < 0.45:
        return rng.choice(pool)
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        m = n
        for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def draw(rng):
    kind = rng.choice(("thermal", "thermal", "elastic", "homog", "homog", "j2", "damage", "plane", "rec"))
    contrast = round(math.exp(rng.uniform(math.log(2.0), math.log(100.0))), 3)
    if rng.random() < 0.3:
        contrast = round(1.0 / contrast, 5)  # the other automatic scheme
    if kind in ("thermal", "elastic"):
        rule = rng.choice(("residual", "residual", "reference"))
        precision = "fp64" if rule == "reference" else rng.choice(("fp64", "fp32_refine"))
        tol = 1e-10 if precision == "fp32_refine" else rng.choice((1e-5, 1e-6, 1e-7))
        n = _length(rng, 24, 160 if kind == "thermal" else 100)
        return {"kind": kind, "n": n, "precision": precision, "rule": rule, "tol": tol, "contrast": contrast}
    if kind == "homog":
        n = _length(rng, 24, 100)
        most = max(1, min(32, 4 * 96 ** 3 // n ** 3))
        rves = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
        return {"kind": kind, "n": n, "precision": "fp32_refine", "tol": 1e-9, "rves": rves}
    if kind == "j2":
        return {"kind": kind, "n": _length(rng, 24, 128), "precision": rng.choice(("fp32", "fp64")), "tol": 1e-4, "increments": rng.randint(1, 3), "strain": 3e-3}
    if kind == "damage":
        return {"kind": kind, "n": _length(rng, 24, 96), "precision": "fp64", "tol": 1e-4, "increments": rng.randint(1, 3), "strain": 3e-3}
    if kind == "plane":
        return {"kind": kind, "n": _length(rng, 64, 1024, ()), "iterations": 25}
    return {"kind": kind, "n": _length(rng, 32, 171, ()), "passes": rng.randint(4, 10)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator().manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _inclusions(n, seed, salt, vf, radius, aspect=1.0, dims=3):
    """Phase map (1 matrix, 0 inclusion) of overlapping periodic ellipsoids (aspect * a, a, a) of random centre and
    direction, as many as give about the volume fraction `vf`."""
    g = _gen(seed, salt)
    size = n ** dims
    one = aspect * (math.pi * radius ** 2 if dims == 2 else 4.0 / 3.0 * math.pi * radius ** 3)
    count = max(1, int(round(-math.log(1.0 - vf) * size / one)))
    centres = torch.rand((count, dims), generator=g, dtype=torch.float64) * n
    direction = torch.randn((count, dims), generator=g, dtype=torch.float64)
    direction /= direction.norm(dim=1, keepdim=True)
    at = torch.arange(n, dtype=torch.float64, device="cuda")
    out = torch.ones((n,) * dims, dtype=torch.int32, device="cuda")
    reach = int(math.ceil(radius * aspect)) + 1
    for c, u in zip(centres.tolist(), direction.tolist()):
        # the box of voxels around the centre, wrapped
        idx, off = [], []
        for d in range(dims):
            if 2 * reach + 1 >= n:
                i = torch.arange(n, device="cuda")
                x = at - c[d]
                x = x - n * torch.round(x / n)
            else:
                k = torch.arange(int(c[d]) - reach, int(c[d]) + reach + 1, device="cuda")
                i, x = k % n, k.double() - c[d]
            idx.append(i)
            off.append(x.reshape([-1 if e == d else 1 for e in range(dims)]))
        along = sum(o * w for o, w in zip(off, u))
        far = sum(o * o for o in off)
        inside = (along / (aspect * radius)) ** 2 + (far - along * along) / radius ** 2 <= 1.0
        view = out[torch.meshgrid(*idx, indexing="ij")]
        out[torch.meshgrid(*idx, indexing="ij")] = torch.where(inside, torch.zeros_like(view), view)
    return out


def _phase(case, seed, salt=0):
    n = case["n"]
    if case["kind"] == "thermal":
        return _inclusions(n, seed, salt, 0.30, max(2.0, 0.062 * n), aspect=3.0)
    if case["kind"] == "plane":
        return _inclusions(n, seed, salt, 0.30, max(3.0, 0.04 * n), dims=2)
    return _inclusions(n, seed, salt, 0.20 if case["kind"] != "homog" else 0.10 + 0.05 * (salt % 5), max(2.0, n / 10.0))


def _materials(case, salt=0):
    """Rows [E, nu, sigma_y, H, n, P, Y0] of phase 0 (inclusion) and 1 (matrix)."""
    if case["kind"] == "j2":
        return np.array([[400e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [70e9, 0.33, 100e6, 1e9, 1.0, 0.0, 1e30]])
    if case["kind"] == "damage":
        return np.array([[20e9, 0.2, 1e30, 0.0, 1.0, 1e-4, 8e2], [3e9, 0.35, 1e30, 0.0, 1.0, 5e-4, 30.0]])
    if case["kind"] == "homog":  # contrasts of the batch workload, a quarter of the RVEs with soft inclusions
        contrast = (5.0, 40.0, 0.05, 15.0)[salt % 4]
        return np.array([[contrast * 3e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [3e9, 0.35, 1e30, 0.0, 1.0, 0.0, 1e30]])
    return np.array([[case["contrast"] * 3e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [3e9, 0.35, 1e30, 0.0, 1.0, 0.0, 1e30]])


PLANE = (3e9, 0.35, 70e9, 0.2)  # E and nu of matrix and inclusion


def _load(case, seed):
    """A load of the path's usual size, its direction from the seed."""
    g = _gen(seed, 77)
    if case["kind"] == "thermal":
        return (torch.rand(3, generator=g, dtype=torch.float64) + 0.5).numpy(), None
    if case["kind"] == "elastic":
        e = (torch.rand(6, generator=g, dtype=torch.float64) + 0.5) * 1e-3
        if _scheme_dual(case):
            e = e * 3e9  # the stress-based scheme is loaded by a stress
        return e.numpy(), np.zeros(6)
    e = np.zeros(6)
    e[0] = case["strain"] * (0.9 + 0.2 * float(torch.rand(1, generator=g)))
    return e, np.array([1.0, 0, 0, 0, 0, 0])


def _scheme_dual(case):
    """Whether the automatic scheme is the stress-based one: the stiffer phase is not the larger one."""
    return case["contrast"] > 1.0


def _spectrum(case, seed):
    """Transform of the isotropic two-point function of the reference's reconstruction example."""
    n = case["n"]
    g = _gen(seed, 5)
    A, Q = 25.0 * (0.9 + 0.2 * float(torch.rand(1, generator=g))), 0.4
    x = torch.arange(n, dtype=torch.float64, device="cuda") - n // 2
    r = torch.sqrt(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2)
    f = torch.where(r == 0, torch.ones_like(r), torch.exp(-r / A) * torch.sin(Q * r) / (Q * torch.where(r == 0, torch.ones_like(r), r)))
    s2 = f * 0.25 + 0.25
    return torch.fft.fftn(torch.fft.ifftshift(s2)).real.contiguous().cpu().numpy().ravel()


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"case": case, "seed": int(seed) & 0xFFFFFFFF}
    if kind in ("thermal", "elastic", "j2", "damage"):
        thermal = kind == "thermal"
        behav = {"j2": m3d.J2, "damage": m3d.DAMAGE}.get(kind, m3d.ELASTIC)
        solver = m3d.Solver(m3d.KIND_THERMAL if thermal else m3d.KIND_MECH, n, n, n, behav, case["precision"])
        phase = _phase(case, seed).cpu().numpy()
        if thermal:
            solver.set_material_thermal(1.0, case["contrast"], phase)
        else:
            solver.set_material_mech(_materials(case), phase)
        solver.set_load(*_load(case, seed))
        s["solver"] = solver
        s["strain"] = _pinned(n ** 3, 3 if thermal else 6)
        if kind == "j2":
            s["plastic"] = _pinned(n ** 3)
        if kind == "damage":
            s["damage"] = _pinned(n ** 3)
    elif kind == "homog":
        solver = m3d.Solver(m3d.KIND_MECH, n, n, n, precision=case["precision"], nrve=case["rves"])
        for r in range(case["rves"]):
            solver.set_material_mech(_materials(case, r), _phase(case, seed, r).cpu().numpy(), rve=r)
        s["solver"] = solver
    elif kind == "plane":
        solver = m3d.Solver2D(n, n)
        solver.material(PLANE, _phase(case, seed).cpu().numpy())
        s["solver"] = solver
        s["strain"], s["stress"] = _pinned(n * n, 3, 2), _pinned(n * n, 3, 2)
    else:
        s["solver"] = m3d.Reconstruction(_spectrum(case, seed), n, n, n)
        s["field"] = _pinned(n ** 3)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, solver = s["case"], s["solver"]
    kind = case["kind"]
    if kind in ("thermal", "elastic"):
        rule = m3d.CRIT_REFERENCE if case["rule"] == "reference" else m3d.CRIT_RESIDUAL
        solver.run(case["tol"], case["tol"], 1, rule)
        solver.field(m3d.FIELD_STRAIN, 0, s["strain"].numpy())
        return {"strain": s["strain"], "means": solver.means()}
    if kind in ("j2", "damage"):
        solver.run(case["tol"], 0.0, case["increments"], m3d.CRIT_RESIDUAL)
        out = {"increments": solver.increments()}
        for name, which in (("strain", m3d.FIELD_STRAIN), ("plastic", m3d.FIELD_EPS_P), ("damage", m3d.FIELD_DAMAGE)):
            if name in s:
                solver.field(which, 0, s[name].numpy())
                out[name] = s[name]
        if case["precision"] == "fp32":  # a program that asks for FP32 goes on in it
            out = {k: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32) for k, v in out.items()}
        return out
    if kind == "homog":
        stiffness, compliance, strains, stresses, _ = solver.homogenize(case["tol"])
        return {"stiffness": stiffness, "compliance": compliance, "strains": strains, "stresses": stresses}
    if kind == "plane":
        solver.set_load([0.005, 0.0, 0.0])  # also puts the fields back to the uniform start
        stiffness, strains, stresses = solver.homogenize(case["iterations"])
        solver.L.m3d2d_get_fields(solver.h, s["strain"].data_ptr(), s["stress"].data_ptr())
        return {"stiffness": stiffness, "strains": strains, "stresses": stresses, "strain": s["strain"], "stress": s["stress"]}
    solver.seed(s["seed"])
    solver.run(case["passes"], 0.8)
    solver.L.m3drec_get_field(solver.h, s["field"].data_ptr())
    return {"field": s["field"], "errors": solver.errors()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sweeps(case):
    """Sweeps to the tolerance at the accelerated scheme's contraction rate."""
    kind = case["kind"]
    if kind in ("j2", "damage"):
        return 100 * case["increments"]  # basic scheme, from its use
    c = 20.0 if kind == "homog" else case["contrast"]
    r = math.sqrt(max(c, 1.0 / c))
    return max(4, math.log(1.0 / case["tol"]) / math.log((r + 1.0) / (r - 1.0)) if r > 1.01 else 4)


def work(case):
    """Per sweep the state is read and written once (in the type the sweeps run in) with the phase ids; the transforms
    are one forward and one inverse real 3-D FFT per component (2.5 log2 V operations a voxel each)."""
    kind, n = case["kind"], case["n"]
    if kind == "plane":
        V, it = n * n, 3 * case["iterations"]
        return {"bytes": it * V * (2 * 48 + 4) + V * 96, "flops": it * V * (3 * 2 * 5 * math.log2(V) + 60)}
    V = n ** 3
    if kind == "rec":
        return {"bytes": case["passes"] * V * (2 * 16 + 8) + 8 * V, "flops": case["passes"] * V * (2 * 5 * math.log2(V) + 20)}
    C = 3 if kind == "thermal" else 6
    entries = 6 * case["rves"] if kind == "homog" else 1
    w = 8 if case["precision"] == "fp64" else 4
    state = 2 * C * w + 1
    if kind == "j2":
        state = 8 * (6 + 6 + 6 + 6 + 1 + 6) + 1  # strain in and out, stress out, the last step's strain, stress and plastic strain
    elif kind == "damage":
        state = 8 * (6 + 6 + 6 + 1 + 1) + 1
    sweeps = _sweeps(case)
    out = 0 if kind == "homog" else 8 * C * V
    return {"bytes": entries * sweeps * V * state + out, "flops": entries * sweeps * V * C * (2 * 2.5 * math.log2(V) + 20)}


# ---------------------------------------------------------------------------
# the same results from plain torch in 64 bits
# ---------------------------------------------------------------------------
def _freq(n, positive_nyquist=False):
    i = torch.arange(n, device="cuda")
    return torch.where(i <= (n // 2 if positive_nyquist else (n - 1) // 2), i, i - n).double()


def _fwd(f):
    return torch.fft.fftn(torch.fft.rfft(f, dim=-1), dim=(-3, -2))


def _bwd(s, n):
    """Complex inverse transforms over x and y, then c2r over z, which ignores the imaginary parts at z = 0 and N/2."""
    s = torch.fft.ifftn(s, dim=(-3, -2))
    s[..., 0] = s[..., 0].real.to(s.dtype)
    if n % 2 == 0:
        s[..., n // 2] = s[..., n // 2].real.to(s.dtype)
    return torch.fft.irfft(s, n=n, dim=-1)


def _xi(n, positive_nyquist=False):
    f = _freq(n, positive_nyquist)
    return f[: n // 2 + 1][None, None, :], f[None, :, None], f[:, None, None]


SHEAR = (1.0, 1.0, 1.0, 2.0, 2.0, 2.0)
PAIRS = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))


def _iso(la, mu):
    C = np.zeros((6, 6))
    C[:3, :3] = la
    C[range(3), range(3)] += 2 * mu
    C[range(3, 6), range(3, 6)] = 2 * mu
    return C


def _pick(v, phase):
    """v[phase] in 64 bits for two numbers v."""
    return torch.where(phase == 0, torch.full_like(phase, v[0], dtype=torch.float64), torch.full_like(phase, v[1], dtype=torch.float64))


def _apply(M, phase, x):
    """M[phase] x for x = [..., C, n, n, n] and one C x C matrix (or number) per phase."""
    if not isinstance(M[0], np.ndarray):
        return _pick(M, phase) * x
    y = [torch.einsum("ab,...bxyz->...axyz", torch.as_tensor(m, device="cuda"), x) for m in M]
    return torch.where(phase == 0, y[0], y[1])


def _green_elastic(t, n, la0, mu0, dual):
    """-Gamma0 t (strain-based) or -Delta0 t (stress-based) of a symmetric tensor field t = [..., 6, modes]."""
    xi = _xi(n)
    q2 = xi[0] ** 2 + xi[1] ** 2 + xi[2] ** 2
    q2 = torch.where(q2 == 0, torch.ones_like(q2), q2)
    T = [[t[..., {(0, 0): 0, (1, 1): 1, (2, 2): 2, (1, 2): 3, (2, 1): 3, (0, 2): 4, (2, 0): 4, (0, 1): 5, (1, 0): 5}[(i, j)], :, :, :]
          for j in range(3)] for i in range(3)]
    u = [sum(T[i][j] * xi[j] for j in range(3)) for i in range(3)]
    s = sum(xi[i] * u[i] for i in range(3))
    out = torch.empty_like(t)
    if not dual:
        a, b = 1.0 / (2 * mu0), (la0 + mu0) / (mu0 * (la0 + 2 * mu0))
        for c, (i, j) in enumerate(PAIRS):
            out[..., c, :, :, :] = -(a * (xi[j] * u[i] + xi[i] * u[j]) / q2 - b * s * xi[i] * xi[j] / q2 ** 2)
    else:
        c1, c2 = 2 * mu0 * (3 * la0 + 2 * mu0) / (la0 + 2 * mu0), 2 * mu0
        tr = T[0][0] + T[1][1] + T[2][2] - s / q2
        for c, (i, j) in enumerate(PAIRS):
            d = 1.0 if i == j else 0.0
            p = d - xi[i] * xi[j] / q2
            out[..., c, :, :, :] = -((c1 - c2) / 2 * p * tr + c2 * (T[i][j] - (xi[i] * u[j] + xi[j] * u[i]) / q2 + s * xi[i] * xi[j] / q2 ** 2))
    return out


def _green_thermal(t, n, k0, dual):
    xi = _xi(n, positive_nyquist=not dual)
    q2 = xi[0] ** 2 + xi[1] ** 2 + xi[2] ** 2
    q2 = torch.where(q2 == 0, torch.ones_like(q2), q2)
    d = sum(xi[i] * t[..., i, :, :, :] for i in range(3)) / q2
    out = torch.empty_like(t)
    for i in range(3):
        out[..., i, :, :, :] = -k0 * (t[..., i, :, :, :] - xi[i] * d) if dual else -xi[i] * d / k0
    return out


def _eq_variable(q, n):
    """The reference's equilibrium variable of a flux (stress) field [C, n, n, n]."""
    C = q.shape[0]
    h = _fwd(q)
    p = h.real ** 2 + h.imag ** 2
    z = _xi(n, positive_nyquist=C == 3)
    w = SHEAR if C == 6 else (1.0, 1.0, 1.0)
    dd = math.sqrt(sum(w[c] * float(p[c, 0, 0, 0]) for c in range(C)))
    s = p[0] * z[0] ** 2 + p[1] * z[1] ** 2 + p[2] * z[2] ** 2
    if C == 6:
        s = s + 2 * p[3] * (z[1] + z[2]) + 2 * p[4] * (z[0] + z[2]) + 2 * p[5] * (z[0] + z[1])
        s = s[:, :, 1:]
    return float(torch.sqrt(torch.abs(s)).sum()) / dd / n ** 3


def _linear(case, phase, E, table, tol, rule="residual"):
    """The accelerated scheme on loads E = [B, C] of one RVE: the primary fields [B, C, n, n, n].  Loads that reach the
    tolerance stop there."""
    P, A, other, flux, green, den = table
    n, B, C = case["n"], len(E), len(E[0])
    E = torch.as_tensor(np.asarray(E), device="cuda")
    V = n ** 3
    w = torch.tensor(SHEAR if C == 6 else (1.0,) * 3, dtype=torch.float64, device="cuda")
    x = E[:, :, None, None, None].expand(B, C, n, n, n).clone()
    norm = torch.sqrt((w * E * E).sum(1))
    live = list(range(B))
    last, eq_last = [float(_apply(other, phase, x[b]).sum()) for b in range(B)], [0.0] * B
    for it in range(1, 2001 if C == 6 else 501):
        y = x[live]
        s = green(_fwd(_apply(P, phase, y)))
        s[..., 0, 0, 0] = (E[live] * V).to(s.dtype)
        d = _bwd(s, n) - y
        y = y + _apply(A, phase, d)
        x[live] = y
        if rule == "residual":
            res = torch.sqrt((w[:, None, None, None] * d * d).sum((1, 2, 3, 4)) / V) / norm[live]
            live = [b for b, r in zip(live, res.tolist()) if not r < tol]
        else:
            b = live[0]
            total, eq = float(_apply(other, phase, y[0]).sum()), _eq_variable(_apply(flux, phase, y[0]) if flux else y[0], n)
            done = it > 1 and abs(eq - eq_last[b]) < tol and abs((total - last[b]) / (V * den * float(E[b].sum()))) < tol
            last[b], eq_last[b] = total, eq
            live = [] if done else live
        if not live:
            break
    return x


def _elastic_table(mat, phase, n):
    """Tables of the elastic scheme that the reference picks, and whether it is the stress-based one."""
    E, nu = mat[:, 0], mat[:, 1]
    mu, la = E / (1 + nu) / 2, nu * E / (1 + nu) / (1 - 2 * nu)
    K = la + 2.0 / 3.0 * mu
    mu0 = math.sqrt(mu.min() * mu.max())
    la0 = math.sqrt(K.min() * K.max()) - 2.0 / 3.0 * mu0
    ones = int((phase != 0).sum())
    vol = (n ** 3 - ones, ones)
    dual = vol[int(np.argmax(mu))] != max(vol)
    Cs = [_iso(la[i], mu[i]) for i in range(2)]
    M = [np.linalg.inv(c) for c in Cs] if dual else Cs
    M0 = np.linalg.inv(_iso(la0, mu0)) if dual else _iso(la0, mu0)
    A = [2 * np.linalg.inv(m + M0) @ M0 for m in M]
    green = lambda t: _green_elastic(t, n, la0, mu0, dual)  # noqa: E731
    return ([m - M0 for m in M], A, M, None if dual else Cs, green, 0.5 * M[0][0, 0] + 0.5 * M[1][0, 0]), dual


def _thermal_table(case, phase):
    n, km, ki = case["n"], 1.0, case["contrast"]
    whole = int((phase != 0).sum()) // n ** 3
    dual = not ((whole >= 0.5 and km > ki) or (whole < 0.5 and km < ki))
    k0 = math.sqrt(km * ki)
    m, m0 = ([1 / ki, 1 / km], 1 / k0) if dual else ([ki, km], k0)
    green = lambda t: _green_thermal(t, n, k0, dual)  # noqa: E731
    return ([v - m0 for v in m], [2 * m0 / (v + m0) for v in m], m, None if dual else m, green, 0.5 * m[0] + 0.5 * m[1]), dual


def _mean(f):
    return f.mean((-3, -2, -1)).cpu().numpy()


def _rows(f):
    """[C, n, n, n] -> [V, C], as the solver hands fields out."""
    return f.reshape(f.shape[0], -1).T.contiguous()


def _exact_linear(case, seed):
    phase = _phase(case, seed)
    if case["kind"] == "thermal":
        table, dual = _thermal_table(case, phase)
    else:
        table, dual = _elastic_table(_materials(case), phase, case["n"])
    tol = case["tol"] * (0.01 if case["precision"] == "fp32_refine" else 1.0)  # refinement: against the converged field
    x = _linear(case, phase, [_load(case, seed)[0]], table, tol, case["rule"])[0]
    other = _apply(table[2], phase, x)
    strain, stress = (other, x) if dual else (x, other)
    return {"strain": _rows(strain), "means": (_mean(strain), _mean(stress))}


def _exact_homog(case, seed):
    found = {k: [] for k in ("stiffness", "compliance", "strains", "stresses")}
    for r in range(case["rves"]):
        phase = _phase(case, seed, r)
        table, dual = _elastic_table(_materials(case, r), phase, case["n"])
        x = _linear(case, phase, np.eye(6) * (1.0e6 if dual else 0.0005), table, case["tol"] * 0.01)
        prim, other = _mean(x), _mean(_apply(table[2], phase, x))  # [load, component]
        e, q = (other, prim) if dual else (prim, other)
        ep, sg = e.T, q  # a column per load case, a row per load case
        if dual:
            S = np.linalg.inv(sg) @ ep
            C = np.linalg.inv(S)
        else:
            C = np.linalg.inv(ep) @ sg
            S = np.linalg.inv(C)
        for k, v in zip(("stiffness", "compliance", "strains", "stresses"), (C, S, ep, sg)):
            found[k].append(v)
    return {k: np.stack(v) if case["rves"] > 1 else v[0].copy() for k, v in found.items()}  # one RVE: the matrices alone


def _mises(s):
    m = (s[0] + s[1] + s[2]) / 3.0
    sd = s.clone()
    sd[:3] -= m
    return math.sqrt(1.5) * torch.sqrt(sum(SHEAR[c] * sd[c] * sd[c] for c in range(6))), sd


def _exact_inelastic(case, seed):
    """Basic scheme with mixed control: J2 return mapping or scalar damage."""
    n, V = case["n"], case["n"] ** 3
    phase, mat = _phase(case, seed), _materials(case)
    E, nu = mat[:, 0], mat[:, 1]
    mu, la = E / (1 + nu) / 2, nu * E / (1 + nu) / (1 - 2 * nu)
    mu0, la0 = (mu.min() + mu.max()) / 2, (la.min() + la.max()) / 2
    Cs = [_iso(la[i], mu[i]) for i in range(2)]
    S0 = np.linalg.inv(_iso(la0, mu0))
    mup, Sy, H, P, Y0 = (_pick(v, phase) for v in (mu, mat[:, 2], mat[:, 3], mat[:, 5], mat[:, 6]))
    load, X0 = _load(case, seed)
    inc = case["increments"]
    dE = load / inc
    dot = lambda a, b: float(sum(SHEAR[c] * a[c] * b[c] for c in range(6)))  # noqa: E731
    eps = torch.as_tensor(dE, device="cuda")[:, None, None, None].expand(6, n, n, n).clone()
    eps_old, sig_old = torch.zeros_like(eps), torch.zeros_like(eps)
    ep = torch.full((n, n, n), 1.236547e-9, dtype=torch.float64, device="cuda")
    dmg = torch.zeros((n, n, n), dtype=torch.float64, device="cuda")
    j2 = case["kind"] == "j2"
    step_form = j2 and case["precision"] == "fp32"  # the FP32 transforms take the load step's stress increment
    norm = math.sqrt(dot(dE, dE))

    def update(eps):
        """stress, plastic multiplier where the yield function is positive (J2), damage"""
        if not j2:
            ce = _apply(Cs, phase, eps)
            Y = torch.sqrt(sum(SHEAR[c] * ce[c] * eps[c] for c in range(6)))
            d = torch.where(Y > Y0, torch.maximum(1 - torch.exp(-P * (Y - Y0)), dmg), dmg)
            return (1 - d) * ce, None, d
        sig = sig_old + _apply(Cs, phase, eps - eps_old)
        seff, sd = _mises(sig)
        phi = seff - Sy - H * ep
        x = torch.where(phi > 0, phi / (3 * mup + H), torch.zeros_like(phi))  # linear hardening: one Newton step
        sig = sig - (1.5 * x / torch.where(phi > 0, seff, torch.ones_like(seff))) * _apply(Cs, phase, sd)
        return sig, x, None

    rows = np.zeros((inc, 9))
    for k in range(inc):
        sig, dp, d = update(eps)
        dmg = dmg if j2 else d
        for _ in range(2000):
            ms, me = _mean(sig), _mean(eps)
            x = S0 @ ms - me
            f = (dE.sum() * (k + 1) + dot(x, X0)) / dot(S0 @ X0, X0)
            Eb = f * (S0 @ X0) - x
            s = _green_elastic(_fwd(sig - sig_old if step_form else sig), n, la0, mu0, False)
            s[:, 0, 0, 0] = torch.as_tensor((Eb - me) * V, device="cuda").to(s.dtype)
            de = _bwd(s, n)
            del s
            eps = eps + de
            res = math.sqrt(float(sum(SHEAR[c] * (de[c] * de[c]).sum() for c in range(6))) / V) / norm
            del de
            sig, dp, d = update(eps)
            dmg = dmg if j2 else d
            if res < case["tol"]:
                break
        rows[k, 0] = float(eps[0].mean())
        rows[k, 1:7] = _mean(sig)
        rows[k, 7] = float(_mises(sig)[0].mean()) if j2 else float(dmg.mean())
        rows[k, 8] = float(ep.mean()) if j2 else 0.0
        if j2:
            ep = ep + dp
            sig_old = sig.clone()
        eps, eps_old = eps + (eps - eps_old), eps  # the next step starts from the extrapolated strain
    out = {"increments": rows, "strain": _rows(eps)}
    if j2:
        out["plastic"] = ep.reshape(-1)
    else:
        out["damage"] = dmg.reshape(-1)
    return out


def _exact_plane(case, seed):
    n, V = case["n"], case["n"] ** 2
    matrix = _phase(case, seed) == 1
    Em, vm, Ei, vi = PLANE
    mum, lam, mui, lai = Em / (1 + vm) / 2, vm * Em / (1 + vm) / (1 - 2 * vm), Ei / (1 + vi) / 2, vi * Ei / (1 + vi) / (1 - 2 * vi)
    iso = lambda la, mu: np.array([[la + 2 * mu, la, 0], [la, la + 2 * mu, 0], [0, 0, 2 * mu]])  # noqa: E731
    Cm, Ci = (torch.as_tensor(iso(la, mu), device="cuda").to(torch.complex128) for la, mu in ((lam, mum), (lai, mui)))
    C0, la0, mu0 = (Cm + Ci) / 2, (lai + lam) / 2, (mui + mum) / 2
    f = _freq(n)
    z = (f[:, None], f[None, :])
    q2 = z[0] ** 2 + z[1] ** 2
    q2 = torch.where(q2 == 0, torch.ones_like(q2), q2)
    a, b = 1 / (4 * mu0), (la0 + mu0) / (mu0 * (la0 + 2 * mu0))
    delta = lambda i, j: 1.0 if i == j else 0.0  # noqa: E731
    pairs = ((0, 0), (1, 1), (0, 1))

    def G(r, c):
        (i, j), (k, h) = pairs[r], pairs[c]
        return a / q2 * (delta(k, i) * z[h] * z[j] + delta(h, i) * z[k] * z[j] + delta(k, j) * z[h] * z[i] + delta(h, j) * z[k] * z[i]) - b * z[i] * z[j] * z[k] * z[h] / q2 ** 2

    # the operator is kept as its upper triangle, so rows read each pair once
    op = [[G(min(r, c), max(r, c)) for c in range(3)] for r in range(3)]
    eps = torch.zeros((3, n, n), dtype=torch.complex128, device="cuda")
    eps[0] = 0.005
    ep, sg, sig = np.zeros((3, 3)), np.zeros((3, 3)), None
    for w in range(3):
        for _ in range(case["iterations"]):
            sig = torch.where(matrix, torch.einsum("ab,bxy->axy", Cm, eps), torch.einsum("ab,bxy->axy", Ci, eps))
            t = torch.fft.fft2(sig - torch.einsum("ab,bxy->axy", C0, eps))
            s = torch.stack([-(op[r][0] * t[0] + op[r][1] * t[1] + 2 * op[r][2] * t[2]) for r in range(3)])
            s[:, 0, 0] = 0
            s[w, 0, 0] = 0.005 * V
            eps = torch.fft.ifft2(s)
        ep[w] = (eps.real.sum((1, 2)) / V).cpu().numpy()
        sg[:, w] = (sig.real.sum((1, 2)) / V).cpu().numpy()
    both = [torch.view_as_real(t.reshape(3, -1).T.contiguous()) for t in (eps, sig)]
    return {"stiffness": np.linalg.inv(ep) @ sg, "strains": ep, "stresses": sg, "strain": both[0], "stress": both[1]}


def _uniform(seed, n):
    """The documented draws of the reconstruction: 2u - 1 from two rounds of the SplitMix64 finaliser."""
    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    with np.errstate(over="ignore"):
        v = mix(mix(np.array([seed], np.uint64) * np.uint64(0x100000001B3)) + np.arange(n, dtype=np.uint64))
    return 2.0 * ((v >> np.uint64(11)).astype(np.float64) / 9007199254740992.0) - 1.0


def _exact_rec(case, seed):
    n, V, beta = case["n"], case["n"] ** 3, 0.8
    amp = torch.sqrt(torch.abs(torch.as_tensor(_spectrum(case, seed), device="cuda").reshape(n, n, n)) * V)
    m = torch.as_tensor((_uniform(int(seed) & 0xFFFFFFFF, V) + 1.0) * 0.5, device="cuda").reshape(n, n, n).to(torch.complex128)
    errors = []
    for _ in range(case["passes"]):  # far fewer than the 100 after which the projection changes
        M = torch.fft.fftn(m)
        errors.append(float(torch.abs(M.abs() - amp).mean()))
        if errors[-1] < 0.1:
            break
        h = torch.fft.ifftn(amp * M / M.abs())
        re, im = h.real, h.imag
        under = re < 0
        re, im = torch.where(under, m.real - beta * re, re), torch.where(under, torch.zeros_like(im), im)
        over = re > 1
        re, im = torch.where(over, m.real - beta * (re - 1), re), torch.where(over, torch.zeros_like(im), im)
        over = re > 1
        re, im = torch.where(over, torch.ones_like(re), re), torch.where(over, torch.zeros_like(im), im)
        m = torch.complex(re, im)
    target, x, tries = float(amp[0, 0, 0]) / V, 0.0, 0
    while True:
        cut = torch.where(m.real < 0.5 - x, 0.0, 1.0).double()
        gap = float(cut.sum()) / V - target
        x = x - 0.001 if gap > 0 else x + 0.001
        if abs(gap) < 0.0001 or tries > 200:
            break
        tries += 1
    return {"field": cut.reshape(-1), "errors": np.array(errors)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("thermal", "elastic"):
        return _exact_linear(case, seed)
    if kind == "homog":
        return _exact_homog(case, seed)
    if kind in ("j2", "damage"):
        return _exact_inelastic(case, seed)
    return _exact_plane(case, seed) if kind == "plane" else _exact_rec(case, seed)
