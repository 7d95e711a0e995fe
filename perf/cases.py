"""Performance cases of the SPM time step: whole passes through the public entry points.

A pass advances a resident run by a few steps with `SPMRun.step` (or `Pool.step`) and reads back what a program
of that kind reads: the particle records, and in some cases a field of the frame.  Sizes are those of the
repository's own workloads (the reference's parity, thermostat, precision, sheared and serving configurations)
and generic ones around them.  `exact` restates the Navier-Stokes and Lees-Edwards steps in 64-bit torch; it
shares no code with the library.  The Electrolyte and squirmer cases run in FP64, where the tolerance against
another FP64 implementation is itself far below single precision, and have no restatement here.
"""
import math

import numpy as np
import torch

from kapsel3_b200 import _native as N
from kapsel3_b200.serve import Pool
from kapsel3_b200.spm import SPMRun, pack_particles, unpack_particles
from kapsel3_b200.udf import EQ_EL, EQ_LE, EQ_NS, SPMConfig

SHEAR_RATE = 1e-3
KBT = 1e-4


def _case(name, kind, nx, ny, nz, colloids, prec, steps, a=4, kbt=False, read="particles", runs=1):
    """nx, ny, nz: grid points; read: "particles" (records after the steps), "exchange" (records uploaded and read
    around every step), "zeta" or "velocity" (records and that field after the steps)."""
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, colloids=colloids, prec=prec, steps=steps, a=a, kbt=kbt, read=read,
             runs=runs)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest run: two colloids under a constant force, looked at after every step
        _case("ns_32_single_step", "ns", 32, 32, 32, 2, "fp64", 1),
        # FP64 drop-in with thermal noise: 200 colloids, trajectory and fields compared every 50 steps
        _case("ns_128_thermostat_fp64", "ns", 128, 128, 128, 200, "fp64", 50, a=5, kbt=True, read="zeta"),
        # the precision form's workload as a coupled program drives it: records in and out every step
        _case("ns_256_exchange_fp32", "ns", 256, 256, 256, 1000, "fp32", 10, a=5, read="exchange"),
        # the same workload, FP64, run freely between looks at the particles
        _case("ns_256_fp64", "ns", 256, 256, 256, 1000, "fp64", 10, a=5),
        # a box that is not a cube with an odd count of colloids, an output frame every 50 steps
        _case("ns_slab_frame_fp32", "ns", 128, 64, 256, 83, "fp32", 50, read="velocity"),
        # the largest grids: an axis of 512 points, fields of 270 MB
        _case("ns_512_fp32", "ns", 512, 256, 256, 1501, "fp32", 4, a=5),
        # sheared suspension with Lees-Edwards boundaries, and the stress line of every look
        _case("le_128_fp32", "le", 128, 128, 128, 400, "fp32", 20),
        _case("le_64_fp64", "le", 64, 64, 64, 47, "fp64", 10, read="zeta"),
        # serving: eight independent runs of one grid size stepped together
        _case("pool_64_fp32", "pool", 64, 64, 64, 75, "fp32", 20, runs=8),
        # charged colloids in salt under a constant field
        _case("el_128_fp64", "el", 128, 128, 128, 50, "fp64", 5, a=5),
        # squirmers with the self-consistent slip iteration
        _case("squirmers_64_fp64", "sq", 64, 64, 64, 50, "fp64", 4, a=5),
    ]


def draw(rng):
    kind = rng.choice(["ns", "ns", "ns", "le", "pool", "el", "sq"])
    top = {"ns": 25, "le": 21, "pool": 18, "el": 21, "sq": 19}[kind]  # log2 of the most grid points
    while True:
        ax = [rng.randint(5, 9 if kind == "ns" else 8) for _ in range(3)]
        if 16 <= sum(ax) <= top and max(ax) - min(ax) <= 3:
            break
    nx, ny, nz = (1 << e for e in ax)
    a = rng.choice([4, 5])
    room = nx * ny * nz / (4.0 / 3.0 * math.pi * (a + 1) ** 3)
    colloids = int(math.exp(rng.uniform(0.0, math.log(max(2.0, min(1500.0, 0.15 * room))))))
    prec = "fp64" if kind in ("el", "sq") else rng.choice(["fp32", "fp64"])
    if prec == "fp64" and sum(ax) == 25:
        prec = "fp32"
    steps = max(1, min(rng.randint(1, 30), 1 << max(0, 27 - sum(ax) - (kind != "ns") * 2)))
    kbt = kind in ("ns", "pool") and rng.random() < 0.3
    read = "particles"
    if kind == "ns" and sum(ax) <= 21:
        read = rng.choice(["particles", "exchange", "zeta" if prec == "fp64" else "velocity"])
    runs = rng.randint(2, 11) if kind == "pool" else 1
    return _case(None, kind, nx, ny, nz, colloids, prec, steps, a=a, kbt=kbt, read=read, runs=runs)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(case):
    e = [int(case[k]).bit_length() - 1 for k in ("nx", "ny", "nz")]
    c = SPMConfig(npx=e[0], npy=e[1], npz=e[2], n_particles=case["colloids"], a=float(case["a"]), a_xi=2.0, dt=0.05,
                  kbt=KBT if case["kbt"] else 0.0, equation=EQ_NS)
    kind = case["kind"]
    if kind == "ns" and case["colloids"] <= 2:
        c.body_force = (1e-3, 0.0, 0.0)
    if kind == "le":
        c.equation, c.shear_rate = EQ_LE, SHEAR_RATE
    if kind == "el":
        c.equation, c.salt, c.valency, c.onsager = EQ_EL, True, (1.0, -1.0), (1.0, 1.0)
        c.dielectric, c.debye_length, c.surface_charge = 1.0, 4.0, -20.0
        c.e_field, c.e_ext, c.dt, c.kbt = "DC", (0.05, 0.0, 0.0), 0.005, 1.0
    if kind == "sq":
        c.janus_axis, c.janus_propulsion, c.dt = "Z", "SQUIRMER", 0.1
        c.slip_vel, c.slip_mode, c.slip_tol, c.slip_iter = 0.015, 1.0, 0.005, 4
    return c


def _particles(case, seed, run=0):
    """Seeded positions without overlap, random orientations, Gaussian velocities."""
    rng = np.random.default_rng([seed, run])
    n, box = case["colloids"], np.array([case["nx"], case["ny"], case["nz"]], float)
    x = np.zeros((n, 3))
    for i in range(n):
        for _ in range(100000):
            c = rng.random(3) * box
            d = x[:i] - c
            d -= np.rint(d / box) * box
            if i == 0 or (d * d).sum(1).min() > (1.05 * 2.0 * case["a"]) ** 2:
                break
        else:
            raise ValueError("no room for %d colloids" % n)
        x[i] = c
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return dict(x=x, v=rng.normal(0.0, 1e-3, (n, 3)), omega=rng.normal(0.0, 1e-4, (n, 3)), q=q)


def _pinned(n):
    t = torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def _prec(case):
    return N.SPM_PREC_FP64 if case["prec"] == "fp64" else N.SPM_PREC_FP32_MIXED


def prepare(case, seed):
    cfg = _config(case)
    n = case["colloids"]
    state = dict(case=case, seed=seed)
    if case["kind"] == "pool":
        pool = Pool(cfg, precision=_prec(case), capacity=case["runs"])
        state["pool"] = pool
        state["runs"] = [pool.admit(cfg, _particles(case, seed, r), mt_seed=r) for r in range(case["runs"])]
        pool.synchronize()
        return state
    run = SPMRun(cfg, precision=_prec(case))
    run.initialize(_particles(case, seed))
    run.synchronize()
    state["run"] = run
    state["rec"] = _pinned(n * N.SPM_PARTICLE_WORDS).reshape(n, N.SPM_PARTICLE_WORDS)
    if case["read"] in ("zeta", "velocity"):
        count = 2 if case["read"] == "zeta" else 3
        state["fields"] = [_pinned(run.nfield) for _ in range(count)]
    if case["read"] == "exchange":
        state["rec"][:] = run.particles_record()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
# what a look at the particles uses: positions, velocities, orientations and the forces of the step just done
SEEN = ("x", "v", "omega", "q", "f_hydro_previous", "torque_hydro_previous", "fr_previous")


def _seen(rec):
    p = unpack_particles(rec)
    return {k: p[k] for k in SEEN}


def run(state):
    case = state["case"]
    if case["kind"] == "pool":
        pool = state["pool"]
        pool.step(case["steps"])
        pool.synchronize()
        return [_seen(pool.particles(r, case["colloids"])) for r in state["runs"]]
    r, rec = state["run"], state["rec"]
    if case["read"] == "exchange":
        for _ in range(case["steps"]):
            N.check(r.L.spm_set_particles(r.h, N.dptr(rec)), "spm_set_particles")
            r.step(1)
            N.check(r.L.spm_get_particles(r.h, N.dptr(rec)), "spm_get_particles")
        return _seen(rec)
    r.step(case["steps"])
    N.check(r.L.spm_get_particles(r.h, N.dptr(rec)), "spm_get_particles")
    out = _seen(rec)
    nx, ny, nz = r.shape
    if case["read"] == "zeta":
        z, dc = state["fields"], np.zeros(3)
        N.check(r.L.spm_get_zeta(r.h, N.dptr(z[0]), N.dptr(z[1]), N.dptr(dc)), "spm_get_zeta")
        out["zeta"] = [f.view(np.complex128).reshape(nx, ny, nz // 2 + 1) for f in z]
    elif case["read"] == "velocity":
        u = state["fields"]
        N.check(r.L.spm_get_velocity(r.h, *[N.dptr(f) for f in u]), "spm_get_velocity")
        out["velocity"] = [f.reshape(nx, ny, -1)[:, :, :nz] for f in u]
    if case["kind"] == "le":
        deg, stress = r.shear_state()
        out["degree_oblique"], out["stress"] = deg, stress[[0, 4, 5, 7]]  # rate, hydrodynamic, Reynolds, apparent
    return out


# ---------------------------------------------------------------------------
# measures
# ---------------------------------------------------------------------------
def work(case):
    """Per step the reduced vorticity (two fields of the retained 2/3 box; FP32 keeps a compensation word) and the
    particle state are read and written once, Electrolyte runs their ion concentrations too; the operations are
    those of the step's real transforms, 2.5 n log2 n each."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells = nx * ny * nz
    box = (2 * ((nx + 2) // 3) - 1) * (2 * ((ny + 2) // 3) - 1) * ((nz + 2) // 3)
    fields = 2 + (2 if case["kind"] == "el" else 0)
    state = box * 16.0 * fields  # 16 bytes: an FP64 complex value, or an FP32 one with its compensation
    if case["kind"] == "le" and case["prec"] == "fp32":
        state /= 2.0
    transforms = {"ns": 14, "pool": 14, "le": 15, "el": 36, "sq": 38}[case["kind"]]
    steps, runs = case["steps"], case["runs"]
    back = case["colloids"] * N.SPM_PARTICLE_WORDS * 8.0
    frame = {"zeta": 2, "velocity": 3}.get(case["read"], 0) * 8.0 * nx * ny * (nz + 2)
    return {"bytes": runs * (steps * (2.0 * state + 2.0 * back) + back + frame),
            "flops": runs * steps * transforms * 2.5 * cells * math.log2(cells)}


def tolerance(case):
    # Measured against the 64-bit restatement: FP64 up to 6e-14 (torques under Lees-Edwards), FP32 up to 3e-6, under
    # Lees-Edwards 3e-5 (the hydrodynamic torque of colloids that hardly turn, a difference of nearly equal sums).
    if case["prec"] == "fp64":
        return {"rel": 1e-11, "max": 1e-8} if case["kind"] in ("el", "sq") else {"rel": 1e-12, "max": 1e-9}
    return {"rel": 1.2e-4, "max": 1e-2} if case["kind"] == "le" else {"rel": 1.2e-5, "max": 1e-3}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
class _Exact:
    """Time_evolution_hydro and Time_evolution_hydro_OBL of spheres at DX = RHO = ETA = 1, density ratio 1."""

    def __init__(self, case, cfg, parts, mt_seed=0):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.le = case["kind"] == "le"
        self.dt, self.kbt, self.bf = cfg.dt, cfg.kbt, cfg.body_force
        self.n3 = n3 = [case["nx"], case["ny"], case["nz"]]
        self.a = float(case["a"])
        t = lambda v: torch.as_tensor(np.asarray(v, float), device=self.dev)  # noqa: E731
        self.L = t(n3)
        self.x, self.v, self.w, self.q = (t(parts[k]).clone() for k in ("x", "v", "omega", "q"))
        self.q = self.q / self.q.norm(dim=1, keepdim=True)
        self.vo, self.wo, self.qo = torch.zeros_like(self.v), torch.zeros_like(self.w), self.q.clone()
        self.fr_prev = torch.zeros_like(self.v)
        self.mdf = torch.zeros_like(self.v)
        mode = lambda n: torch.tensor([i - n if i > n // 2 else i for i in range(n)], device=self.dev)  # noqa: E731
        KX, KY = mode(n3[0])[:, None, None], mode(n3[1])[None, :, None]
        KZ = torch.arange(n3[2] // 2 + 1, device=self.dev)[None, None, :]
        self.nzx, self.nzy, self.nzz = KX != 0, KY != 0, KZ != 0
        trn = [(n + 2) // 3 for n in n3]
        self.keep = (KX.abs() < trn[0]) & (KY.abs() < trn[1]) & (KZ < trn[2])
        self.k = [2 * math.pi / n * K.double() for n, K in zip(n3, (KX, KY, KZ))]
        h = int(case["a"]) + 4
        r = torch.arange(-h, h + 1, device=self.dev)
        c = torch.cartesian_prod(r, r, r)
        self.cells = c[(c.double() ** 2).sum(1).sqrt() < self.a + 1.0 + 1.7321]
        self.rng = np.random.RandomState(mt_seed)
        self.gam, self.rate, self.ts = 0.0, 0.0, 0
        self.metric()
        shape = (n3[0], n3[1], n3[2] // 2 + 1)
        self.zeta = [torch.zeros(shape, dtype=torch.complex128, device=self.dev) for _ in range(2)]
        self.dc = torch.zeros(3, dtype=torch.float64, device=self.dev)
        # initial projection of the particles' velocities
        flat, rv, dist, sg, _ = self.stencil()
        self.phi(flat, dist)
        up = self.scatter(flat, self.surface(rv, sg) * self.weight(flat, dist)[..., None])
        uk = self.project([self.fft(f) * self.keep for f in up], False)
        self.zeta = self.curl_reduce(uk, False)
        if self.le:
            self.v[:, 0] = 0.0
            self.w[:, 2] = 0.0

    def metric(self):
        k2 = self.k[0] ** 2 + (self.k[1] - self.k[0] * self.gam) ** 2 + self.k[2] ** 2
        self.k2, self.ik2 = k2, torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)), 0.0)

    def fft(self, f):
        return torch.fft.rfftn(f)

    def ifft(self, f):
        return torch.fft.irfftn(f, s=self.n3)

    def lower(self, v):  # contravariant -> covariant
        g = self.gam
        return [v[0] + g * v[1], g * v[0] + (1 + g * g) * v[1], v[2]]

    def cross_ik(self, v, s=None):
        kx, ky, kz = self.k if s is None else [k * s for k in self.k]
        return [1j * (ky * v[2] - kz * v[1]), 1j * (kz * v[0] - kx * v[2]), 1j * (kx * v[1] - ky * v[0])]

    def omega_of(self, z, obl):
        kx, ky, kz = self.k
        safe = lambda k: torch.where(k != 0, k, torch.ones_like(k))  # noqa: E731
        first = -(ky * z[0] + kz * z[1]) / safe(kx)
        if obl:
            rest = [torch.where(self.nzz, z[1], z[0]), torch.where(self.nzz, z[0], 0.0),
                    torch.where(self.nzz, -(ky / safe(kz)) * z[0], z[1])]
        else:
            rest = [torch.where(self.nzy, z[1], z[0]), torch.where(self.nzy, -(kz / safe(ky)) * z[0], z[1]),
                    torch.where(self.nzy, z[0], 0.0)]
        return [torch.where(self.nzx, f, r) for f, r in zip((first, z[0], z[1]), rest)]

    def reduce(self, om, obl):
        if obl:
            rest = [torch.where(self.nzz, om[1], om[0]), torch.where(self.nzz, om[0], om[2])]
        else:
            rest = [torch.where(self.nzy, om[2], om[0]), torch.where(self.nzy, om[0], om[1])]
        return [torch.where(self.nzx, f, r) for f, r in zip((om[1], om[2]), rest)]

    def curl_reduce(self, u, obl):
        return self.reduce(self.cross_ik(self.lower(u) if obl else u), obl)

    def u_of(self, z, obl):
        om = self.omega_of(z, obl)
        u = self.cross_ik(self.lower(om) if obl else om, self.ik2)
        for d in range(3):
            u[d][0, 0, 0] = self.dc[d]
        return u

    def project(self, u, obl):
        kx, ky, kz = self.k
        g = self.gam if obl else 0.0
        d = self.ik2 * (u[0] * kx + u[1] * ky + u[2] * kz)
        return [u[0] - d * ((1 + g * g) * kx - g * ky), u[1] - d * (ky - g * kx), u[2] - d * kz]

    @staticmethod
    def near(a):
        return torch.where(a >= 0, torch.trunc(a + 0.5), torch.trunc(a - 0.5))

    def stencil(self):
        n3, c = self.n3, self.cells[None]
        xi = torch.trunc(self.x).long()
        res = self.x - xi
        raw = xi[:, None, :] + c
        m = torch.stack([(raw[..., d] + n3[d]) % n3[d] for d in range(3)], -1)
        r = c.double() - res[:, None, :]
        if not self.le:
            d = self.x[:, None, :] - m
            d = d - self.near(d / self.L) * self.L
            return (m[..., 0] * n3[1] + m[..., 1]) * n3[2] + m[..., 2], r, (d * d).sum(-1).sqrt(), None, m[..., 1]
        sg = torch.sign(raw[..., 1] - m[..., 1]).double()
        fx = torch.fmod(xi[:, None, 0] - sg * self.gam * n3[1] + res[:, None, 0] + c[..., 0] + 4 * n3[0], float(n3[0]))
        m0 = fx.long()
        r = torch.stack([c[..., 0] - (fx - m0), r[..., 1], r[..., 2]], -1)
        y = self.x[:, None, 1] - m[..., 1]
        y1 = y - self.near(y / n3[1]) * n3[1]
        s = torch.sign(torch.trunc(y - y1))
        x1 = self.x[:, None, 0] - (m0 + s * self.gam * n3[1])
        x1 = x1 - self.near(x1 / n3[0]) * n3[0]
        z1 = self.x[:, None, 2] - m[..., 2]
        z1 = z1 - self.near(z1 / n3[2]) * n3[2]
        dist = (x1 * x1 + y1 * y1 + z1 * z1).sqrt()
        return (m0 * n3[1] + m[..., 1]) * n3[2] + m[..., 2], r, dist, sg, m[..., 1]

    def profile(self, d):
        def H(y):
            return torch.where(y > 0, torch.exp(-1.0 / torch.where(y > 0, y, torch.ones_like(y)) ** 2), 0.0)
        h = H(self.a + 1.0 - d)
        return h / (h + H(d - self.a + 1.0))

    def phi(self, flat, dist):
        s = torch.zeros(self.n3[0] * self.n3[1] * self.n3[2], dtype=torch.float64, device=self.dev)
        self.phi_sum = s.index_add_(0, flat.reshape(-1), self.profile(dist).reshape(-1))

    def weight(self, flat, dist):
        return self.profile(dist) / self.phi_sum[flat].clamp(min=1.0)

    def surface(self, r, sg):
        vs = self.v[:, None, :] + torch.linalg.cross(self.w[:, None, :].expand_as(r), r)
        if sg is not None:
            vs = torch.stack([vs[..., 0] - sg * self.rate * self.n3[1], vs[..., 1], vs[..., 2]], -1)
        return vs

    def scatter(self, flat, val):
        out = []
        for d in range(3):
            f = torch.zeros(self.phi_sum.numel(), dtype=torch.float64, device=self.dev)
            out.append(f.index_add_(0, flat.reshape(-1), val[..., d].reshape(-1)).view(self.n3))
        return out

    def pair_forces(self):
        sigma = 2.0 * self.a
        d = self.x[None, :, :] - self.x[:, None, :]  # x_j - x_i
        if self.le:
            sigma = min((sigma + 2.0) / 2.0 ** (1.0 / 6.0), sigma)
            y = d[..., 1]
            y1 = y - self.near(y / self.n3[1]) * self.n3[1]
            s = torch.sign(torch.trunc(y - y1))
            x1 = d[..., 0] - s * self.gam * self.n3[1]
            x1 = x1 - self.near(x1 / self.n3[0]) * self.n3[0]
            d = torch.stack([x1, y1, d[..., 2] - self.near(d[..., 2] / self.n3[2]) * self.n3[2]], -1)
            mult = 1.0
        else:
            d = d - self.near(d / self.L) * self.L
            mult = torch.ones(d.shape[:2], dtype=torch.float64, device=self.dev)
            for ax in range(3):  # cells of 16 points; with fewer than three an axis' neighbour cell counts again
                lc = self.n3[ax] // 16
                m = torch.trunc(self.x[:, ax] / 16).long()
                mult *= sum(((m + o) % lc)[:, None] == m[None, :] for o in (-1, 0, 1)).double()
        r = (d * d).sum(-1).sqrt()
        ok = (r < sigma * 2.0 ** (1.0 / 6.0)) & ~torch.eye(len(r), dtype=torch.bool, device=self.dev)
        rr = torch.where(ok, r, torch.ones_like(r))
        s6 = (sigma / rr) ** 6
        mag = torch.where(ok, 24.0 / (rr * rr) * (2.0 * s6 * s6 - s6), 0.0) * mult
        pair = -mag[..., None] * d
        lj = 0.5 * (pair[..., 0] * d[..., 1]).sum()
        return pair.sum(1) + torch.tensor(self.bf, dtype=torch.float64, device=self.dev), lj

    def noise(self):
        n, got, buf = len(self.x), [], []
        while len(got) < 3 * n:
            x1, x2 = (2.0 * (float(self.rng.randint(0, 1 << 32, dtype=np.uint32)) + 0.5) / 4294967296.0 - 1.0
                      for _ in range(2))
            rsq = x1 * x1 + x2 * x2
            if 0.0 < rsq < 1.0:
                f = math.sqrt(-2.0 * math.log(rsq) / rsq)
                got.append((f * x1, f * x2))
        buf = torch.tensor(got, dtype=torch.float64, device=self.dev).view(n, 6)
        mass = 4.0 / 3.0 * math.pi * self.a ** 3
        sv = 1.439 * math.sqrt(6.0 * math.pi * self.a * self.dt * self.kbt)
        so = 1.22 * math.sqrt(8.0 * math.pi * self.a ** 3 * self.dt * self.kbt)
        self.v = self.v + buf[:, :3] * sv / mass
        self.w = self.w + buf[:, 3:] * so / (0.4 * mass * self.a ** 2)

    def move(self):
        euler, dt = self.ts == 0, self.dt
        self.x = self.x + (dt * self.v if euler else 0.5 * dt * (3.0 * self.v - self.vo))
        n3 = self.n3
        if self.le:
            y = torch.fmod(self.x[:, 1] + n3[1], float(n3[1]))
            s = torch.sign(torch.trunc(self.x[:, 1] - y))
            self.x = torch.stack([torch.fmod(self.x[:, 0] - s * self.gam * n3[1] + n3[0], float(n3[0])), y,
                                  torch.fmod(self.x[:, 2] + n3[2], float(n3[2]))], 1)
            self.v[:, 0] -= s * self.rate * n3[1]
            self.vo[:, 0] -= s * self.rate * n3[1]
        else:
            self.x = torch.fmod(self.x + self.L, self.L)

        def rate(q, w):
            s, v = q[:, :1], q[:, 1:]
            return 0.5 * torch.cat([-(w * v).sum(1, keepdim=True), s * w + torch.linalg.cross(w, v)], 1)
        dq = rate(self.q, self.w)
        q = self.q + dt * dq if euler else self.q + 1.5 * dt * dq - 0.5 * dt * rate(self.qo, self.wo)
        self.qo, self.q = self.q, q / q.norm(dim=1, keepdim=True)

    def shift(self, f, to_oblique):
        """Linear interpolation between the oblique and the orthogonal grid, one y plane at a time."""
        nx, ny, _ = self.n3
        out = torch.empty_like(f)
        for j in range(ny):
            dj = j - ny // 2
            sign = float(np.sign(dj if self.gam >= 0 else -dj))
            base = float(int(sign * self.gam * dj)) * sign
            if to_oblique:
                io, al = base, (self.gam * dj - base) * sign
                out[:, :, j] = (1 - al) * f[:, :, j].roll(-int(io), 1) + al * f[:, :, j].roll(-int(io + sign), 1)
            else:
                io = base + sign
                al = (io - self.gam * dj) * sign
                out[:, :, j] = ((1 - al) * f[:, :, j] + al * f[:, :, j].roll(-int(sign), 1)).roll(int(io), 1)
        return out

    def step(self):
        le, n3, dt = self.le, self.n3, self.dt
        zeta = [z * self.keep for z in self.zeta]
        uk = self.u_of(zeta, le)
        u = [self.ifft(f) for f in uk]
        if le:
            om = self.omega_of(zeta, True)
            for f in om:
                f[0, 0, 0] = 1j * f[0, 0, 0].imag
            om = [self.ifft(f) for f in om]
            p = [self.fft(u[1] * om[2] - u[2] * om[1]) - 2.0 * self.rate * uk[1],
                 self.fft(u[2] * om[0] - u[0] * om[2]) - 2.0 * self.rate * self.gam * uk[1],
                 self.fft(u[0] * om[1] - u[1] * om[0])]
            force = self.reduce(self.cross_ik(p), True)
        else:
            p = [self.fft(f) for f in (u[1] * u[2], u[2] * u[0], u[0] * u[1], (u[1] - u[2]) * (u[1] + u[2]),
                                       (u[2] - u[0]) * (u[2] + u[0]))]
            k1, k2, k3 = self.k
            a2 = -p[4] - p[3]
            force = self.reduce(
                [-(k2 * k3 * p[3] + (k3 * k3 - k2 * k2) * p[0] + k3 * k1 * p[2] - k1 * k2 * p[1]),
                 -(k3 * k1 * p[4] + (k1 * k1 - k3 * k3) * p[1] + k1 * k2 * p[0] - k2 * k3 * p[2]),
                 -(k1 * k2 * a2 + (k2 * k2 - k1 * k1) * p[2] + k2 * k3 * p[1] - k3 * k1 * p[0])], False)
        e = torch.expm1(-dt * self.k2)
        zeta = [(z + e * (z - self.ik2 * f)) * self.keep for z, f in zip(zeta, force)]
        del p, force, e
        self.dc = torch.zeros_like(self.dc)
        u = torch.stack([self.ifft(f) for f in self.u_of(zeta, le)])
        ug = u
        if le:
            self.rate = SHEAR_RATE
            self.gam += self.rate * dt
            assert self.gam < n3[0] / n3[1]  # a pass ends before the grid is sheared by one box
            self.metric()
            ug = self.shift(u, False)
            ug[0] += self.gam * ug[1]
            ug[0] += self.rate * (torch.arange(n3[1], device=self.dev).double() - n3[1] / 2.0)[None, :, None]
            ip, im, g = u[0].roll(-1, 0), u[0].roll(1, 0), self.gam
            above = 0.5 * ((1 - g) * ip.roll(-1, 1) + (1 + g) * im.roll(-1, 1))
            below = 0.5 * ((1 - g) * im.roll(1, 1) + (1 + g) * ip.roll(1, 1))
            self.rate += float((above - below).sum()) * 0.5 / u[0].numel()
        self.move()
        flat, r, dist, sg, m1 = self.stencil()
        self.phi(flat, dist)
        w = self.weight(flat, (r * r).sum(-1).sqrt() if le else dist)
        d = (self.surface(r, sg) - torch.stack([f.reshape(-1)[flat] for f in ug], -1)) * w[..., None]
        f, tq = d.sum(1), torch.linalg.cross(r, d).sum(1)
        stress = {}
        if le:
            ry = m1 + sg * n3[1]
            vol, trace = w.sum(1), (w * (r * r).sum(-1)).sum(1) * (2.0 / 3.0)
            turn = -(tq[:, 1, None] * r[..., 2] - tq[:, 2, None] * r[..., 1]) / trace[:, None]
            new = (d[..., 0] * ry).sum() + (-(f[:, 0] / vol) * (ry * w).sum(1)).sum() + (turn * ry * w).sum()
            dy = (torch.arange(n3[1], device=self.dev) - n3[1] // 2).double()[None, :, None]
            cells = n3[0] * n3[1] * n3[2]
            stress = dict(hydro=-float(new) / cells / dt,
                          reynolds=-float(((ug[0] - self.rate * dy) * ug[1]).sum()) / cells)
        self.f, self.tq = -f / dt, -tq / dt
        fr, lj = self.pair_forces()
        mass = 4.0 / 3.0 * math.pi * self.a ** 3
        self.vo, self.wo = self.v.clone(), self.w.clone()
        if self.ts == 0:
            self.v = self.v + dt / mass * (self.f + fr)
            self.w = self.w + dt / (0.4 * mass * self.a ** 2) * self.tq
        else:
            self.v = self.v + 0.5 * dt / mass * (2.0 * self.f + fr + self.fr_prev)
            self.w = self.w + dt / (0.4 * mass * self.a ** 2) * self.tq
        self.fr_prev = fr
        if self.kbt > 0.0:
            self.noise()
        up = self.scatter(flat, self.surface(r, sg) * self.weight(flat, dist)[..., None])
        f = torch.stack(up) - self.phi_sum.clamp(max=1.0).view(n3) * ug
        if le:
            f = self.shift(f, True)
            f[0] -= self.gam * f[1]
            uk = [self.fft(c) for c in u + f]
            self.dc = torch.stack([c[0, 0, 0].real for c in uk])
            self.zeta = self.curl_reduce(self.project(uk, True), True)
            self.stress = [self.rate, stress["hydro"], stress["reynolds"],
                           stress["hydro"] + stress["reynolds"] + float(lj) / f[0].numel() + self.rate]
        else:
            fk = [self.fft(c) * self.keep for c in f]
            self.dc = self.dc + torch.stack([c[0, 0, 0].real for c in fk])
            uk = [a + b for a, b in zip(self.u_of(zeta, False), self.project(fk, False))]
            self.zeta = self.curl_reduce(uk, False)
        self.ts += 1

    def seen(self):
        v = (self.x, self.v, self.w, self.q, self.f, self.tq, self.fr_prev)
        return {k: t.cpu().numpy() for k, t in zip(SEEN, v)}


def exact(case, seed):
    if case["kind"] in ("el", "sq"):
        return None
    cfg = _config(case)
    out = []
    for r in range(case["runs"]):
        e = _Exact(case, cfg, _particles(case, seed, r), mt_seed=r if case["kind"] == "pool" else 0)
        for _ in range(case["steps"]):
            e.step()
        out.append(e.seen())
    if case["kind"] == "pool":
        return out
    got = out[0]
    if case["read"] == "zeta":
        got["zeta"] = [z.cpu().numpy() for z in e.zeta]
    elif case["read"] == "velocity":
        got["velocity"] = [e.ifft(f).cpu().numpy() for f in e.u_of(e.zeta, False)]
    if case["kind"] == "le":
        got["degree_oblique"], got["stress"] = e.gam, np.array(e.stress)
    return got
