"""The calls that programs on this framework spend their time in, as timing cases.

A case is one of these kinds (``kind``):

``md``     a batch of replicas on a ``Context``, advanced ``steps`` velocity-Verlet
           steps by ``Context.run`` (graph-launched), then the state, the
           energies and -- where the run records it -- n(q,t) read back: one
           chunk of a production run.
``mixed``  the same over replicas of different N, coupling, screening and mesh.
``force``  ``yukawa_p3m_ord6.force_pot`` on host arrays.
``update`` ``velocity_verlet_p3m_ord6.update`` on host arrays.
``green``  ``yukawa_gf_opt.gf_opt``: the influence function of a new parameter set.
``sqw``    ``s_of_q_w_avg.s_of_q_w_avg_mat``: S(q,w) of recorded n(q,t) series.

Units are the reference's (lengths in a_ws, time in 1/omega_p, T = 1/Gamma).
Particles start near a bcc lattice (thermal displacements and Maxwell
velocities, in random memory order), as in a strongly coupled plasma: the
framework's own random start needs hundreds of steps before it looks like
one. The FP32 path's results hold single-precision numbers in double arrays;
a case of that path hands them on in single precision.

``exact`` evaluates the same formulas in plain FP64 torch: a cell-list pair
sum, the order-6 charge assignment, the full complex FFT chain.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "md-force-routines_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import s_of_q_w_avg  # noqa: E402
import velocity_verlet_p3m_ord6  # noqa: E402
import yukawa_gf_opt  # noqa: E402
import yukawa_p3m_ord6  # noqa: E402
from p3m_b200 import FP32, FP64, MODE_NVE, MODE_THERMOSTAT, Context, Replica  # noqa: E402

yukawa_p3m_ord6.VERBOSE = False  # the energy line of every call: off in timed loops

DT, AF, UF, KF = 0.1, 1.0 / 3.0, 1.0, 1.5
ORDER, ALIAS = 6, 3
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def box(n):
    return (4.0 * math.pi * n / 3.0) ** (1.0 / 3.0)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest system of the tests, thermostat phase: latency and launches
        dict(name="md-2e3-m32-thermostat", kind="md", n=2000, replicas=1, gamma=100.0, kappa=2.0,
             alpha=0.6, rc=6.0, mesh=32, precision="fp32", mode="thermostat", steps=40, nq=0,
             skin=-1.0, prune=0.0),
        # one 1e4-particle replica, production with n(q,t): what the reference's driver runs
        dict(name="md-1e4-m64-nqt", kind="md", n=10000, replicas=1, gamma=100.0, kappa=2.0,
             alpha=0.6, rc=6.0, mesh=64, precision="fp32", mode="nve", steps=40, nq=32, skin=0.8,
             prune=0.0),
        # the same on the plain FP64 path, default shapes
        dict(name="md-1e4-m64-fp64", kind="md", n=10000, replicas=1, gamma=100.0, kappa=2.0,
             alpha=0.6, rc=6.0, mesh=64, precision="fp64", mode="nve", steps=20, nq=0, skin=-1.0,
             prune=0.0),
        # the batched ensemble of the benchmark, with the shapes its tuner installs
        dict(name="md-20x1e4-m64-nqt", kind="md", n=10000, replicas=20, gamma=100.0, kappa=2.0,
             alpha=0.6, rc=6.0, mesh=64, precision="fp32", mode="nve", steps=20, nq=32, skin=1.1,
             prune=0.3),
        # one larger replica, multi-pass FFTs
        dict(name="md-1e5-m128-nqt", kind="md", n=100000, replicas=1, gamma=50.0, kappa=1.0,
             alpha=0.5, rc=7.0, mesh=128, precision="fp32", mode="nve", steps=20, nq=32, skin=0.8,
             prune=0.0),
        # uneven ensemble (N 2e3 .. 5e4, meshes 32 .. 128), equilibration, default shapes
        dict(name="mixed-12-thermostat", kind="mixed", systems=12, system_seed=100,
             precision="fp32", mode="thermostat", steps=20, nq=0, skin=-1.0, prune=0.0),
        # the largest replica
        dict(name="md-1e6-m256", kind="md", n=1000000, replicas=1, gamma=100.0, kappa=2.0,
             alpha=0.6, rc=6.0, mesh=256, precision="fp32", mode="nve", steps=10, nq=0, skin=1.1,
             prune=0.3),
        # drop-in calls on host arrays, FP64 (the reference's arithmetic)
        dict(name="force-1e4-m64", kind="force", n=10000, gamma=100.0, kappa=2.0, alpha=0.6,
             rc=6.0, mesh=64),
        dict(name="update-1999-m32", kind="update", n=1999, gamma=100.0, kappa=2.0, alpha=0.6,
             rc=6.0, mesh=32),
        # a new parameter set's influence function
        dict(name="green-m64", kind="green", n=10000, kappa=2.0, alpha=0.6, mesh=64),
        # spectra of four recorded runs
        dict(name="sqw-4x4096", kind="sqw", n=10000, runs=4, nt=4096, nq=6),
    ]


def _mesh_for(n):
    # spacings of 0.4 .. 0.9 a_ws, as the hand-set and picked parameters have
    for m in (32, 64, 128):
        if box(n) / m <= 0.75:
            return m
    return 256


def _ewald(n, mesh):
    # the PM error of order 6 is near 1e-6 at alpha h = 0.33, the PP one at
    # alpha rc = 3.6; three cells of rc fit the box
    alpha = 0.33 * mesh / box(n)
    return alpha, min(3.6 / alpha, box(n) / 3.0 * (1.0 - 1e-9))


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["md"] * 7 + ["fp64"] * 2 + ["mixed"] * 2 + ["force", "update", "green", "sqw"])
    gamma, kappa = _log_uniform(rng, 10.0, 200.0), rng.uniform(0.5, 3.0)
    if kind == "md":
        total = _log_uniform(rng, 2000.0, 400000.0)
        reps = rng.choice([1, 1, rng.randint(2, 20)])
        n = max(1000, int(total / reps))
        mesh = _mesh_for(n)
        alpha, rc = _ewald(n, mesh)
        skin, prune = rng.choice([(-1.0, 0.0), (0.8, 0.0), (1.1, 0.3)])
        if min(skin, box(n) / 3.0 - rc) <= prune:
            skin, prune = -1.0, 0.0
        return dict(kind="md", n=n, replicas=reps, gamma=gamma, kappa=kappa, alpha=alpha, rc=rc,
                    mesh=mesh, precision="fp32", mode=rng.choice(["nve", "nve", "thermostat"]),
                    steps=rng.randint(8, 24), nq=rng.choice([0, rng.randint(1, 32)]), skin=skin,
                    prune=prune)
    if kind == "fp64":
        n = int(_log_uniform(rng, 1000.0, 60000.0))
        mesh = _mesh_for(n)
        alpha, rc = _ewald(n, mesh)
        return dict(kind="md", n=n, replicas=1, gamma=gamma, kappa=kappa, alpha=alpha, rc=rc,
                    mesh=mesh, precision="fp64", mode=rng.choice(["nve", "thermostat"]),
                    steps=rng.randint(8, 20), nq=rng.choice([0, 16]), skin=-1.0, prune=0.0)
    if kind == "mixed":
        return dict(kind="mixed", systems=rng.randint(3, 16), system_seed=rng.randint(1, 10000),
                    precision="fp32", mode=rng.choice(["nve", "thermostat"]),
                    steps=rng.randint(8, 20), nq=rng.choice([0, 16]), skin=-1.0, prune=0.0)
    if kind == "green":
        n = int(_log_uniform(rng, 2000.0, 200000.0))
        mesh = rng.choice([32, 64, 96, 128])
        return dict(kind="green", n=n, kappa=kappa, alpha=0.33 * mesh / box(n), mesh=mesh)
    if kind == "sqw":
        return dict(kind="sqw", n=10000, runs=rng.randint(1, 8),
                    nt=rng.choice([1024, 2048, 4096, rng.randint(600, 5000)]), nq=rng.randint(1, 8))
    n = int(_log_uniform(rng, 1000.0, 60000.0 if kind == "force" else 20000.0))
    mesh = _mesh_for(n)
    alpha, rc = _ewald(n, mesh)
    return dict(kind=kind, n=n, gamma=gamma, kappa=kappa, alpha=alpha, rc=rc, mesh=mesh)


def _systems(case):
    """[(N, gamma, kappa, alpha, rc, mesh)] of a case's replicas."""
    if case["kind"] != "mixed":
        one = (case["n"], case.get("gamma", 100.0), case["kappa"], case["alpha"], case.get("rc", 0.0),
               case["mesh"])
        return [one] * case.get("replicas", 1)
    rng = np.random.default_rng(case["system_seed"])
    out = []
    for _ in range(case["systems"]):
        n = int(round(math.exp(rng.uniform(math.log(2000.0), math.log(50000.0)))))
        gamma = math.exp(rng.uniform(math.log(10.0), math.log(200.0)))
        kappa = rng.uniform(0.5, 3.0)
        mesh = _mesh_for(n)
        out.append((n, gamma, kappa) + _ewald(n, mesh) + (mesh,))
    return out


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _lattice_cells(n):
    """(a, b, c) with 2 a b c >= n, near-cubic, fewest vacancies."""
    e = max(1, int(round((n / 2.0) ** (1.0 / 3.0))))
    best = None
    for a in range(max(1, e - 1), e + 3):
        for b in range(a, e + 3):
            for c in range(b, e + 3):
                if 2 * a * b * c >= n and (best is None or a * b * c < best[0]):
                    best = (a * b * c, (a, b, c))
    return best[1]


def _start(n, gamma, rng):
    """Positions and velocities of one replica."""
    L = box(n)
    a, b, c = _lattice_cells(n)
    i, j, k = np.meshgrid(np.arange(a), np.arange(b), np.arange(c), indexing="ij")
    corner = np.stack([i.ravel() / a, j.ravel() / b, k.ravel() / c], axis=1)
    sites = np.concatenate([corner, corner + np.array([0.5 / a, 0.5 / b, 0.5 / c])])
    pos = sites[rng.permutation(len(sites))[:n]] * L
    pos += rng.random(3) * L + rng.normal(0.0, min(0.3, 0.12 * math.sqrt(100.0 / gamma)), (n, 3))
    pos -= L * np.floor(pos / L)
    pos[pos >= L] = 0.0
    vel = rng.normal(0.0, math.sqrt(1.0 / gamma / 3.0), (n, 3))
    return np.ascontiguousarray(pos), vel - vel.mean(axis=0)


def _inputs(case, seed):
    rng = np.random.default_rng([int(seed), 20])
    s = [_start(n, gamma, rng) for n, gamma, *_ in _systems(case)]
    return np.concatenate([p for p, _ in s]), np.concatenate([v for _, v in s])


def _series(case, seed):
    """n(q,t) of `runs` runs at 3 nq wave numbers: damped oscillations and noise."""
    rng = np.random.default_rng([int(seed), 21])
    t = np.arange(case["nt"])[:, None, None] * DT
    out = np.empty((case["runs"], case["nt"], 3 * case["nq"], 3), dtype=np.complex128)
    for r in range(case["runs"]):
        w = rng.uniform(0.2, 1.2, (1, 3 * case["nq"], 3))
        ph = rng.uniform(0.0, 2 * np.pi, (1, 3 * case["nq"], 3))
        noise = rng.normal(size=(2,) + out.shape[1:])
        out[r] = 40.0 * np.exp(-0.002 * t) * np.cos(w * t + ph) + 5.0 * (noise[0] + 1j * noise[1])
    return out


def _scan(case, seed):
    """(kappa, alpha) of one point of a parameter scan around the case's."""
    rng = np.random.default_rng([int(seed), 23])
    return case["kappa"] * rng.uniform(0.98, 1.02), case["alpha"] * rng.uniform(0.98, 1.02)


def _pinned(n):
    t = torch.empty((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "green":
        return {"case": case, "param": _scan(case, seed)}
    if kind == "sqw":
        a = _series(case, seed)
        return {"case": case, "series": a, "out": np.zeros((case["runs"], case["nq"], case["nt"]))}
    pos, vel = _inputs(case, seed)
    if kind in ("force", "update"):
        n, L, M = case["n"], box(case["n"]), case["mesh"]
        G, kv = _green_plan(case["kappa"], case["alpha"], M, L)
        s = {"case": case, "pos": pos, "vel": vel, "Z": np.ones(n), "Lv": np.full(3, L),
             "G": G, "kx": kv.reshape(1, M), "ky": kv.reshape(M, 1), "kz": kv.reshape(M, 1, 1),
             "acc": np.zeros((n, 3)), "acc_s": np.zeros((n, 3)), "acc_f": np.zeros((n, 3)),
             "rho": np.zeros((M, M, M)), "E": [np.zeros(n) for _ in range(3)]}
        if kind == "update":
            s["acc"] = np.random.default_rng([int(seed), 22]).normal(0.0, 0.05, (n, 3))
        return s
    # a context with its graphs captured, its lists' plan set and the state on the device
    f32 = case["precision"] == "fp32"
    reps = [Replica(N=n, L=box(n), kappa=kappa, alpha=alpha, rc=rc, M=mesh, dt=DT,
                    T_desired=1.0 / gamma, af=AF, uf=UF, kf=KF)
            for n, gamma, kappa, alpha, rc, mesh in _systems(case)]
    ctx = Context(reps, precision=FP32 if f32 else FP64)
    if case["skin"] >= 0.0:
        ctx.set_tuning(skin=case["skin"], prune_buf=case["prune"])
    if case["nq"]:
        ctx.set_nqt(np.arange(1, case["nq"] + 1, dtype=np.float64), 64)
    s = {"case": case, "ctx": ctx, "f32": f32, "out": [_pinned(len(pos)) for _ in range(3)],
         "mode": MODE_THERMOSTAT if case["mode"] == "thermostat" else MODE_NVE}
    ctx.set_state_all(pos, vel)
    ctx.init_forces()
    ctx.run(9, s["mode"], record_nqt=case["nq"] > 0)
    ctx.set_state_all(pos, vel)
    ctx.init_forces()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _run_md(s):
    c, ctx = s["case"], s["ctx"]
    ctx.run(c["steps"], s["mode"], record_nqt=c["nq"] > 0, sync=False)
    pos, vel, acc = ctx.get_state_all(*s["out"])
    e = ctx.energies(c["steps"])
    out = {"pos": pos, "vel": vel, "acc": acc, "energies": e}
    if c["nq"]:
        out["nqt"] = np.stack([ctx.get_nqt(r, c["nq"], c["steps"]) for r in range(len(ctx.replicas))])
    if not s["f32"]:
        return {k: torch.from_numpy(v) for k, v in out.items()}
    return {k: torch.from_numpy(v).to(torch.complex64 if np.iscomplexobj(v) else torch.float32)
            for k, v in out.items()}


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("md", "mixed"):
        return _run_md(s)
    if kind == "green":
        M, L = c["mesh"], box(c["n"])
        h = L / M
        G, kx, ky, kz, a_pm = yukawa_gf_opt.gf_opt(*s["param"], ORDER, ALIAS, ALIAS, ALIAS, M, M, M,
                                                   h, h, h, L, L, L)
        return {"G": G, "A_pm": np.array([a_pm])}
    if kind == "sqw":
        return s_of_q_w_avg.s_of_q_w_avg_mat(s["series"], c["nq"], s["out"], c["runs"],
                                             float(c["n"]), DT, c["nt"] * DT)
    n, M = c["n"], c["mesh"]
    L = float(s["Lv"][0])
    h = L / M
    mesh = (s["G"], s["kx"], s["ky"], s["kz"], M, M, M, h, h, h, L, L, L, ORDER, ALIAS, ALIAS, ALIAS)
    scratch = (s["acc_s"], s["acc_f"], s["rho"], *s["E"])
    if kind == "force":
        U, acc = yukawa_p3m_ord6.force_pot(c["kappa"], c["alpha"], n, c["rc"], s["Lv"], AF, UF,
                                           s["pos"], s["acc"], s["Z"], *mesh, *scratch)
        return {"U": np.array([U]), "acc": acc}
    pos, vel, acc, U = velocity_verlet_p3m_ord6.update(
        s["pos"], s["vel"], s["acc"], DT, 1, c["kappa"], n, 3, s["Lv"], s["Lv"], np.zeros(3),
        c["alpha"], c["rc"], AF, UF, s["Z"], *mesh, *scratch)
    return {"pos": pos, "vel": vel, "acc": acc, "U": np.array([U])}


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def work(case):
    """The mesh stages' arrays and the particle state, each written and read
    once per step, and the pairs (48 operations), transforms and stencils."""
    kind = case["kind"]
    if kind == "green":
        m3 = case["mesh"] ** 3
        return {"bytes": 8.0 * m3, "flops": 343.0 * 12 * m3}
    if kind == "sqw":
        series = 3.0 * case["runs"] * case["nq"] * case["nt"]
        return {"bytes": 16.0 * series + 8.0 * series / 3, "flops": 5.0 * series * math.log2(case["nt"])}
    b = f = 0.0
    word = 4.0 if case.get("precision") == "fp32" else 8.0
    steps = case.get("steps", 1)
    for n, _, _, _, rc, mesh in _systems(case):
        m3 = float(mesh) ** 3
        b += 16.5 * word * m3 + (96.0 + 6 * word) * n
        f += n * rc ** 3 / 2 * 48 + 4 * 2.5 * m3 * math.log2(m3) + n * 216 * 8.0
        f += n * 3.0 * 8 * case.get("nq", 0)
    return {"bytes": b * steps, "flops": f * steps}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _green(kappa, alpha, M, L):
    """Optimal influence function (FFT order) and the sum A_pm."""
    dev = DEVICE
    h = L / M
    i = torch.arange(M, device=dev, dtype=torch.float64)
    s = torch.where(i < (M + 1) // 2, i, i - M)
    k = 2 * math.pi * s / L
    m = torch.arange(-ALIAS, ALIAS + 1, device=dev, dtype=torch.float64)
    km = 2 * math.pi * (s[:, None] + m * M) / L
    u2 = torch.sinc(0.5 * km * h / math.pi) ** (2 * ORDER)
    dot = k[:, None] * km
    num = torch.zeros((M, M, M), dtype=torch.float64, device=dev)
    den = torch.zeros_like(num)
    ax = lambda v, d: v.reshape([M if j == d else 1 for j in range(3)])  # noqa: E731
    for a in range(2 * ALIAS + 1):
        for b in range(2 * ALIAS + 1):
            for c in range(2 * ALIAS + 1):
                U = ax(u2[:, a], 0) * ax(u2[:, b], 1) * ax(u2[:, c], 2)
                q = ax(km[:, a] ** 2, 0) + ax(km[:, b] ** 2, 1) + ax(km[:, c] ** 2, 2) + kappa ** 2
                d = ax(dot[:, a], 0) + ax(dot[:, b], 1) + ax(dot[:, c], 2)
                num += U * d * (4 * math.pi * torch.exp(-0.25 * q / alpha ** 2) / q)
                den += U
    ksq = ax(k ** 2, 0) + ax(k ** 2, 1) + ax(k ** 2, 2)
    ksq[0, 0, 0] = 1.0
    G = num / (den ** 2 * ksq)
    A = num ** 2 / (den ** 2 * ksq)
    G[0, 0, 0] = 0.0
    A[0, 0, 0] = 0.0
    return G, float(A.sum()), k


@functools.lru_cache(maxsize=4)
def _green_plan(kappa, alpha, M, L):
    """The influence function a user's program keeps: host array in the
    shifted layout, and its wave numbers."""
    G, _, k = _green(kappa, alpha, M, L)
    return np.ascontiguousarray(torch.fft.fftshift(G).cpu().numpy()), torch.fft.fftshift(k).cpu().numpy()


def _pp(pos, L, kappa, alpha, rc):
    """Pair forces and energy: cells of at least rc, all 27 neighbours."""
    n, dev = len(pos), pos.device
    nc = int(L / rc)
    ci = (pos / (L / nc)).long().clamp(0, nc - 1)
    cell = ci[:, 0] + nc * (ci[:, 1] + nc * ci[:, 2])
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=nc ** 3)
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    table = torch.full((nc ** 3, cap), -1, dtype=torch.long, device=dev)
    table[cell[order], torch.arange(n, device=dev) - start[cell[order]]] = order
    acc = torch.zeros_like(pos)
    U = torch.zeros((), dtype=torch.float64, device=dev)
    span = max(1, int(2.5e7 / (cap * cap)))
    cz, cy, cx = torch.meshgrid(*[torch.arange(nc, device=dev)] * 3, indexing="ij")
    cx, cy, cz = cx.ravel(), cy.ravel(), cz.ravel()
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                nb = (cx + dx) % nc + nc * ((cy + dy) % nc + nc * ((cz + dz) % nc))
                for c0 in range(0, nc ** 3, span):
                    i, j = table[c0:c0 + span, :, None], table[nb[c0:c0 + span]][:, None, :]
                    d = pos[i.clamp(min=0)] - pos[j.clamp(min=0)]
                    d -= L * torch.round(d / L)
                    r2 = (d * d).sum(-1)
                    ok = (r2 < rc * rc) & (i >= 0) & (j >= 0) & (i != j)
                    d, r, i = d[ok], torch.sqrt(r2[ok]), i.expand_as(ok)[ok]
                    ep = torch.exp(kappa * r) * torch.erfc(alpha * r + 0.5 * kappa / alpha)
                    em = torch.exp(-kappa * r) * torch.erfc(alpha * r - 0.5 * kappa / alpha)
                    gs = torch.exp(-(alpha * r) ** 2 - (0.5 * kappa / alpha) ** 2)
                    U += (0.25 * (ep + em) / r).sum()
                    f = 0.5 * (ep * (1 - kappa * r) + em * (1 + kappa * r)) / r ** 2
                    f = f + 2 * alpha / math.sqrt(math.pi) * gs / r
                    acc.index_add_(0, i, (f / r)[:, None] * d)
    return U, acc


def _weights(x):
    c = [[1, -10, 40, -80, 80, -32], [237, -750, 840, -240, -240, 160],
         [1682, -1540, -880, 1120, 160, -320], [1682, 1540, -880, -1120, 160, 320],
         [237, 750, 840, 240, -240, -160], [1, 10, 40, 80, 80, 32]]
    out = []
    for row in c:
        w = torch.zeros_like(x)
        for v in reversed(row):
            w = w * x + v
        out.append(w / 3840.0)
    return out


def _pm(pos, L, M, green):
    G, _, k = green
    h = L / M
    span = 60000  # particles whose 216 nodes are held at once

    def nodes():
        for p0 in range(0, len(pos), span):
            p = pos[p0:p0 + span]
            base = torch.floor(p / h)
            w = [torch.stack(_weights((p[:, d] - (base[:, d] + 0.5) * h) / h), 1) for d in range(3)]
            i = [(base[:, d].long()[:, None] + torch.arange(6, device=p.device)) % M for d in range(3)]
            at = (i[2][:, :, None, None] * M + i[1][:, None, :, None]) * M + i[0][:, None, None, :]
            v = w[2][:, :, None, None] * w[1][:, None, :, None] * w[0][:, None, None, :]
            yield p0, at.reshape(len(p), 216), v.reshape(len(p), 216)

    rho = torch.zeros(M ** 3, dtype=torch.float64, device=pos.device)
    for _, at, v in nodes():
        rho.index_add_(0, at.reshape(-1), v.reshape(-1))
    rk = torch.fft.fftn(rho.reshape(M, M, M))
    U = 0.5 * (rk.abs() ** 2 * G).sum() / L ** 3
    phi = G * rk
    shape = [(1, 1, M), (1, M, 1), (M, 1, 1)]
    E = [(torch.fft.ifftn(-1j * k.reshape(shape[d]) * phi).real * (M / L) ** 3).reshape(-1)
         for d in range(3)]
    acc = torch.empty_like(pos)
    for p0, at, v in nodes():
        for d in range(3):
            acc[p0:p0 + span, d] = (v * E[d][at]).sum(1)
    return U, acc


def _force(pos, system, green):
    n, _, kappa, alpha, rc, M = system
    L = box(n)
    Us, a = _pp(pos, L, kappa, alpha, rc)
    Uf, b = _pm(pos, L, M, green)
    return float(UF * (Us + Uf - n * alpha / math.sqrt(math.pi))), AF * (a + b)


def _step(pos, vel, acc, system, green):
    L = box(len(pos))
    vel = vel + 0.5 * acc * DT
    pos = pos + vel * DT
    pos = torch.where(pos > L, pos - L, pos)
    pos = torch.where(pos < 0.0, pos + L, pos)
    U, acc = _force(pos, system, green)
    return pos, vel + 0.5 * acc * DT, acc, U


def _too_long(case):
    # pair candidates of the cell lists and mesh points, per second on one GPU
    t = 0.0
    for n, _, _, _, rc, mesh in _systems(case):
        cell = box(n) / int(box(n) / rc)
        t += n * 27 * cell ** 3 * 0.24 * 2.5 / 4e9 + n * 216 * 8 / 2e10 + mesh ** 3 / 5e9 + 0.012
    return t * (case.get("steps", 0) + 1) > 18.0


def exact(case, seed):
    kind = case["kind"]
    if kind == "green":
        G, a_pm, _ = _green(*_scan(case, seed), case["mesh"], box(case["n"]))
        return {"G": torch.fft.fftshift(G).cpu(), "A_pm": np.array([a_pm])}
    if kind == "sqw":
        a = torch.from_numpy(_series(case, seed)[:, :, ::3, :])
        S = (torch.fft.fft(a, dim=1) * DT).abs() ** 2 / (case["n"] * case["nt"] * DT)
        return S.mean(-1).permute(0, 2, 1).contiguous()
    if _too_long(case):
        return None
    pos, vel = (torch.from_numpy(v).to(DEVICE) for v in _inputs(case, seed))
    if kind in ("force", "update"):
        system = _systems(case)[0]
        G = _green(case["kappa"], case["alpha"], case["mesh"], box(case["n"]))
        if kind == "force":
            U, acc = _force(pos, system, G)
            return {"U": np.array([U]), "acc": acc.cpu()}
        acc = np.random.default_rng([int(seed), 22]).normal(0.0, 0.05, (case["n"], 3))
        pos, vel, acc, U = _step(pos, vel, torch.from_numpy(acc).to(DEVICE), system, G)
        return {"pos": pos.cpu(), "vel": vel.cpu(), "acc": acc.cpu(), "U": np.array([U])}
    nq, steps = case["nq"], case["steps"]
    outs, first = [], 0
    for system in _systems(case):
        n, gamma = system[:2]
        p, v = pos[first:first + n], vel[first:first + n]
        first += n
        G = _green(system[2], system[3], system[5], box(n))
        _, a = _force(p, system, G)
        rows, series = [], []
        for _ in range(steps):
            p, v, a, U = _step(p, v, a, system, G)
            T = float((v * v).sum()) / n
            fact = math.sqrt(1.0 / gamma / T) if case["mode"] == "thermostat" else 1.0
            v = v * fact
            rows.append([U, KF * T * n, T, fact])
            if nq:
                m = torch.arange(1, nq + 1, device=p.device, dtype=torch.float64)
                ph = 2 * math.pi / box(n) * m[:, None] * p.T[:, None, :]
                series.append(torch.complex(torch.cos(ph).sum(-1), -torch.sin(ph).sum(-1)).T)
        outs.append((p, v, a, np.array(rows), torch.stack(series).cpu() if nq else None))
    out = {k: torch.cat([o[j] for o in outs]).cpu() for j, k in enumerate(("pos", "vel", "acc"))}
    out["energies"] = np.stack([o[3] for o in outs], axis=1)
    if nq:
        out["nqt"] = torch.stack([o[4] for o in outs])
    return out
