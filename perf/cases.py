"""What is timed: the calls that programs built on this framework spend their time in.

A case is one call (or one MD step) of a public entry point on a box of rigid or flexible water:

  md      one step of a captured RigidMD (kick, drift, force call with the induced-dipole solve, kick)
  pimd    one step of a captured PIMD (the beads are a batch of the force field)
  host    pgm_compute_host of an MD engine that owns the coordinates on the host
  point   PGMForceField.compute from an empty induction state (a single point, launched directly)
  field   PGMForceField.field of charges and dipoles (polarizability and response calculations)
  train   one optimiser step of the message-passing guess on a whole frame

The boxes are lattices of `side`^3 pGM3P-25 waters at the density of water, jittered, every molecule
turned to the best of a few trial orientations among its neighbours (a liquid-like start).
`exact` restates the same quantities in float64 with plain torch.
"""

import ctypes
import math

import numpy as np
import torch

from pgm_jax_b200 import _lib
from pgm_jax_b200.forcefield import MDSettings, PGMForceField, elec_cutoff_settings
from pgm_jax_b200.learned import EMAX, GRAPH_CUTOFF, MPNN_SHAPES, SIGMA, MPNNModel
from pgm_jax_b200.md import RigidMD
from pgm_jax_b200.pimd import PIMD
from pgm_jax_b200.systems import Molecule, System

SPACING = 0.3104  # nm between lattice sites: 0.997 g/cm^3
KE, KB, HBAR = 138.935458, 0.0083144626181532, 0.0635077993  # kJ/mol nm e^-2, kJ/mol/K, kJ/mol ps
DT = 1e-3  # ps
WARM = 5  # steps before a timed step: the predictors extrapolate from four
FRAMES = 64  # host: frames of the periodic trajectory

# pGM3P-25 water (O, H, H): e, nm, nm^3, e nm, kJ/mol, amu
Q = (-2.04056220, 1.02028110, 1.02028110)
RADIUS = (0.0605150752, 0.0536231183, 0.0536231183)
ALPHA = (1.11765163e-3, 0.329630770e-3, 0.329630770e-3)
COV = ((0, 1, -0.0191201350), (0, 2, -0.0191201350), (1, 0, 0.00858770326), (2, 0, 0.00858770326))
LJ_A, LJ_B = 5.81935564e5, 5.94825035e2  # kcal A^12/mol, kcal A^6/mol
RMIN_HALF = ((2.0 * LJ_A / LJ_B) ** (1.0 / 6.0) / 20.0, 0.0, 0.0)
SQRT_EPS = (math.sqrt(LJ_B * LJ_B / (4.0 * LJ_A) * 4.184), 0.0, 0.0)
MASS = (16.0, 1.008, 1.008)
# q-TIP4P/F intramolecular term of flexible water: D, alpha, r, k_theta, theta
BOND = (116.09 * 4.184, 22.87, 0.09419, 87.85 * 4.184, math.radians(107.4))


def _case(name, kind, side, **options):
    c = {"kind": kind, "side": side, "systems": 1, "precision": "mixed", "tol": 1e-5, "grid": 0, "predictor": "mu4", "local": 0,
         "elec_cutoff": 0.0, "skew": False}
    c.update(options)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a single point of a small triclinic cell in double precision: parameter fits, validation
        _case("point_64_fp64", "point", 4, precision="double", tol=1e-8, skew=True),
        # the reference's everyday benchmark box, in both precisions
        _case("md_512", "md", 8, grid=48),
        _case("md_512_fp64", "md", 8, grid=48, precision="double"),
        # the 4,096-water benchmark at the tight tolerance, Jacobi preconditioner
        _case("md_4096", "md", 16, grid=96, tol=1e-6),
        # the same box with the shorter electrostatics cutoff (split rows)
        _case("md_4096_split", "md", 16, elec_cutoff=0.7),
        # a box of no special size with the default mesh spacing (108^3)
        _case("md_19683", "md", 27),
        # the headline: 32,768 waters, 192^3, learned guess, local preconditioner
        _case("md_32768_nn", "md", 32, grid=192, tol=1e-6, predictor="nn", local=1),
        # replicas and uneven boxes in one batch: systems of side 7, 8, 9, repeated
        _case("batch_24", "md", 8, systems=24, local=1),
        # path integrals: 32 beads of 512 flexible waters
        _case("pimd_32x512", "pimd", 8, systems=32),
        # an MD engine on the host calling the C ABI
        _case("host_4096", "host", 16, grid=96, tol=1e-6, local=1),
        # fields at given dipoles, in double precision
        _case("field_1728_fp64", "field", 12, precision="double"),
        # training the learned guess
        _case("train_4096", "train", 16),
    ]


def draw(rng):
    kind = rng.choice(["md", "md", "md", "host", "point", "field", "pimd", "train"])
    hi = {"md": 26, "host": 24, "point": 18, "field": 20, "pimd": 8, "train": 20}[kind]
    lo = 5 if kind in ("point", "field", "pimd") else 7
    side = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    o = {"seed": rng.randrange(1000), "tol": rng.choice([1e-5, 1e-6])}
    if kind in ("md", "point", "field") and side <= 14 and rng.random() < 0.4:
        o["precision"] = "double"
    if kind in ("md", "host"):
        o["predictor"] = rng.choice(["mu4", "mu4", "mu3", "mu1"])
        o["local"] = rng.choice([0, 1])
    if kind == "md" and side >= 8 and rng.random() < 0.25:
        o["elec_cutoff"] = 0.7
    if kind == "md" and side <= 9:
        o["systems"] = rng.choice([1, 1, 4, 9, 16])
    if kind == "pimd":
        o["systems"] = rng.randint(4, 32)
    if kind in ("point", "field"):
        o["skew"] = rng.random() < 0.5
    return _case(None, kind, side, **o)


# ----------------------------------------------------------------------------- inputs
def _sides(case):
    """Lattice sides of the batch's systems (pimd: the beads share one)."""
    n = case["systems"]
    return [case["side"]] if n == 1 or case["kind"] == "pimd" else [case["side"] + k % 3 - 1 for k in range(n)]


def _box(case, side):
    a = side * SPACING
    return np.array([[a, 0, 0], [0.2 * a, a, 0], [-0.2 * a, 0.25 * a, a]]) if case["skew"] else np.eye(3) * a


def _images(d, H):
    """d (..., 3) less its lattice vectors, by sequential rounding along c, b, a."""
    for c in (2, 1, 0):
        d = d - torch.round(d[..., c:c + 1] / H[c, c]) * H[c]
    return d


def _rotations(n, gen):
    w, x, y, z = torch.nn.functional.normalize(torch.randn(n, 4, generator=gen, dtype=torch.float64), dim=1).cuda().unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                        1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                        1 - 2 * (x * x + y * y)], 1).view(n, 3, 3)


def _water_box(side, H, seed):
    """Positions (3 side^3, 3), float64 on the GPU."""
    gen = torch.Generator()
    gen.manual_seed(seed)
    n, H = side**3, torch.tensor(H, device="cuda")
    t = math.radians(104.52 / 2)
    w = torch.tensor([[0, 0, 0], [math.sin(t), math.cos(t), 0], [-math.sin(t), math.cos(t), 0]], dtype=torch.float64, device="cuda") * 0.09572
    w = w - w.mean(0)
    k = torch.arange(n, device="cuda")
    site = torch.stack([k // side**2, k // side % side, k % side], 1)
    centre = (site.double() + 0.5) / side @ H + 0.01 * torch.randn(n, 3, generator=gen, dtype=torch.float64).cuda()
    mol = w @ _rotations(n, gen).transpose(1, 2)  # (n, 3 atoms, 3)
    step = torch.cartesian_prod(*[torch.arange(-1, 2, device="cuda")] * 3)
    step = step[(step != 0).any(1)]
    q = torch.tensor(Q, dtype=torch.float64, device="cuda")
    for sweep in range(2):
        for colour in range(8):
            m = k[(site % 2 * torch.tensor([4, 2, 1], device="cuda")).sum(1) == colour]
            nb = ((site[m][:, None] + step) % side * torch.tensor([side**2, side, 1], device="cuda")).sum(-1)
            x = (_images(centre[nb] - centre[m][:, None], H)[:, :, None] + mol[nb]).flatten(1, 2)  # neighbours' atoms
            trial = torch.cat([mol[m][None]] + [(w @ _rotations(len(m), gen).transpose(1, 2))[None] for _ in range(12)])
            e = sum((q[a] * q.repeat(26) / (x - trial[:, :, a, None]).norm(dim=-1)).sum(-1) for a in range(3))
            mol[m] = trial[e.argmin(0), torch.arange(len(m), device="cuda")]
    return (centre[:, None] + mol).view(-1, 3)


def _settings(case):
    small = min(_sides(case)) * SPACING < 1.85  # the cutoff is at most half the box
    o = {"cutoff": 0.6, "ewald_beta": 6.0, "pme_spacing": 0.06} if small else {}
    if case["elec_cutoff"]:
        o.update(elec_cutoff_settings(case["elec_cutoff"]))
    if case["grid"]:
        o["pme_grid"] = (case["grid"],) * 3
    return MDSettings(precision=case["precision"], dipole_tol=case["tol"], max_iter=100, predictor=case["predictor"],
                      local_niter=case["local"], **o)


def _inputs(case, seed):
    """Positions and velocities per system (numpy), boxes."""
    seed = 1000003 * seed + case.get("seed", 0)
    boxes = [_box(case, s) for s in _sides(case)]
    pos = [_water_box(s, H, seed + k).cpu().numpy() for k, (s, H) in enumerate(zip(_sides(case), boxes))]
    rng = np.random.default_rng(seed)
    vel = []
    for x in pos:  # rigid-body velocities at 298 K: a translation and a turn of every molecule
        n, m = len(x) // 3, np.array(MASS)
        y = x.reshape(n, 3, 3)
        c = (m[:, None] * y).sum(1, keepdims=True) / m.sum()
        v = rng.normal(scale=math.sqrt(KB * 298 / m.sum()), size=(n, 1, 3))
        vel.append((v - v.mean(0) + np.cross(rng.normal(scale=14.0, size=(n, 1, 3)), y - c)).reshape(-1, 3))
    return pos, vel, boxes


def _system(n_mol):
    m = Molecule("WAT", ["O", "H", "H"], Q, RADIUS, ALPHA, list(COV), RMIN_HALF, SQRT_EPS, MASS)
    return System([m] * n_mol)


def _train_inputs(case, seed):
    """A frame of the learned guess (graph of a water box, features of its scales) and weights in mid-training."""
    pos = _water_box(case["side"], _box(case, case["side"]), 1000003 * seed + case.get("seed", 0))
    n, H = len(pos), torch.tensor(_box(case, case["side"]), device="cuda")
    i, j = _pair_list(pos, H, GRAPH_CUTOFF)
    i, j = torch.cat([i, j]), torch.cat([j, i])
    order = torch.argsort(i * n + j)
    i, j = i[order], j[order]
    counts = torch.bincount(i, minlength=n)
    slot = torch.arange(len(i), device="cuda") - (counts.cumsum(0) - counts)[i]
    edges = torch.zeros(n, EMAX, 4, device="cuda")
    edges[i, slot, :3] = _images(pos[i] - pos[j], H).float()
    edges[i, slot, 3] = j.int().view(torch.float32)
    gen = torch.Generator()
    gen.manual_seed(seed)
    normal = lambda *s: torch.randn(*s, generator=gen).cuda()  # noqa: E731
    frame = {"inv": normal(n, 16), "vec": 0.02 * normal(n, 15, 3), "edges": edges, "counts": counts.int(), "target": 1e-4 * normal(n, 3)}
    return frame, torch.cat([(normal(*s) * (0.5 / math.sqrt(s[-1]) if len(s) > 1 else 0.1)).flatten() for s in MPNN_SHAPES])


def _trajectory(pos, seed):
    """A smooth periodic trajectory around pos: every molecule swings about its place at thermal speeds."""
    rng = np.random.default_rng(seed)
    n, t = len(pos) // 3, 2 * np.pi * np.arange(FRAMES)[:, None, None] / FRAMES
    a = rng.normal(scale=math.sqrt(KB * 298 / sum(MASS)) * DT * FRAMES / (2 * np.pi), size=(n, 3))
    return pos + np.repeat(np.sin(t + rng.uniform(0, 2 * np.pi, size=(n, 3))) * a, 3, axis=1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        frame, w = _train_inputs(case, seed)
        return {"kind": kind, "frame": frame, "model": MPNNModel(w.cpu().numpy())}
    pos, vel, boxes = _inputs(case, seed)
    systems = [_system(len(x) // 3) for x in pos]
    if kind == "pimd":
        md = PIMD(systems[0], pos[0], boxes[0], _settings(case), beads=case["systems"], dt_fs=1e3 * DT / 2, mode="rpmd", seed=seed)
    else:
        ff = PGMForceField(systems, boxes, _settings(case))
    if kind == "md":
        md = RigidMD(ff, np.concatenate(pos), np.stack(boxes), dt_fs=1e3 * DT, velocities=np.concatenate(vel))
        if case["predictor"] == "nn":
            MPNNModel().install(ff)
    if kind in ("md", "pimd"):
        for _ in range(WARM):
            md.step()
        md.capture()
        return {"kind": kind, "md": md}
    if kind == "host":
        pin = lambda *s: torch.zeros(s, dtype=torch.float64).pin_memory()  # noqa: E731
        s = {"kind": kind, "ff": ff, "at": 0, "frames": torch.from_numpy(_trajectory(pos[0], seed)).pin_memory(), "box": pin(3, 3),
             "energy": pin(3), "forces": pin(ff.n, 3)}
        s["box"].copy_(torch.from_numpy(boxes[0]))
        for _ in range(WARM):
            run(s)
        return s
    x, H = torch.from_numpy(pos[0]).cuda(), torch.from_numpy(boxes[0]).cuda()
    return {"kind": kind, "ff": ff, "pos": x, "box": H, "d": torch.from_numpy(_dipoles(len(x), seed)).cuda()}


def _dipoles(n, seed):
    return np.random.default_rng(seed).normal(scale=0.02, size=(n, 3))


def run(state):
    kind = state["kind"]
    if kind in ("md", "pimd"):
        md, st = state["md"], torch.cuda.current_stream()
        md.stream.wait_stream(st)  # the step's results are read on the caller's stream
        md.run(1)
        st.wait_stream(md.stream)
        return {"pos": md.pos if kind == "md" else md.q, "mom": md.mom if kind == "md" else md.p, "forces": md.forces, "mu": md.ind.mu}
    if kind == "host":
        ff, p = state["ff"], lambda t: ctypes.c_void_p(t.data_ptr())
        out = _lib.PgmOutputs(state["energy"].data_ptr(), state["forces"].data_ptr())
        _lib.check(_lib.load().pgm_compute_host(ff._h, p(state["frames"][state["at"] % FRAMES]), p(state["box"]), None, ctypes.byref(out)))
        state["at"] += 1
        return {"forces": state["forces"]}
    if kind == "point":
        r = state["ff"].compute(state["pos"], state["box"])
        out = {"forces": r.forces, "mu": r.induction.mu}
        if state["ff"].s.precision == "double":  # energies and virial are sums whose mixed-precision rounding is chance
            out.update(energy=r.energy["total"], elec=r.energy["elec"], vdw=r.energy["vdw"], virial=r.virial)
        return out
    if kind == "field":
        return state["ff"].field(state["pos"], state["box"], state["d"])
    m, f = state["model"], state["frame"]
    loss = m.loss_grad(f, 1.0 / (f["inv"].shape[0] * SIGMA**2))
    m.adam()
    return {"loss": loss, "w": m.w, "m": m.m, "v": m.v}


def work(case):
    n = 3 * sum(s**3 for s in _sides(case)) * (case["systems"] if case["kind"] == "pimd" else 1)
    if case["kind"] == "train":
        params = sum(math.prod(s) for s in MPNN_SHAPES)
        return {"bytes": n * (4 * (16 + 45 + 3) + 16 * 52) + 7 * 4 * params, "flops": 3.0 * n * (2 * params + 52 * 2 * (2 * 128 + 30))}
    s = _settings(case)
    rho = 3 / SPACING**3
    half = 0.5 * n * 4 / 3 * math.pi * rho * (s.elec_cutoff or s.cutoff) ** 3
    K = case["grid"] / case["side"] / SPACING if case["grid"] else 1 / s.pme_spacing  # mesh points per nm
    mesh = n / rho * K**3
    sweeps = {"field": 1, "point": 15}.get(case["kind"], 2 + (8 if case["tol"] < 1e-5 else 6))
    flops = half * (80 + 40 * sweeps + 80) + (sweeps + 1) * (2 * 5 * mesh * math.log2(max(mesh, 2)) / 2 + n * 216 * 20)
    return {"bytes": n * {"field": 72, "point": 72, "host": 48 + 2 * 120}.get(case["kind"], 2 * 32 + 48 + 2 * 120), "flops": flops}


# ----------------------------------------------------------------------------- float64 values
def _pair_list(pos, H, rc):
    """All pairs i < j closer than rc (minimum image)."""
    out = []
    for a in range(0, len(pos), 1024):
        d2 = (_images(pos[a:a + 1024, None] - pos[None, a:], H) ** 2).sum(-1)
        i, j = torch.nonzero(d2 < rc * rc, as_tuple=True)
        out.append(torch.stack([i, j])[:, i < j] + a)
    return torch.cat(out, 1)


def _screened(a, r):
    """B_0, B_1, B_2 of erf(a r) / r (B_n+1 = -B_n' / r)."""
    c = 2 / math.sqrt(math.pi) * a * torch.exp(-(a * r) ** 2)
    b0 = torch.erf(a * r) / r
    b1 = (b0 - c) / r**2
    return b0, b1, (3 * b1 - 2 * a * a * c) / r**2


def _tile(v, n):
    return torch.tensor(v, dtype=torch.float64, device="cuda").repeat(n // 3)


class _Model:
    """Energy, field and converged dipoles of one water box in float64 (smooth PME on the case's mesh)."""

    def __init__(self, n, s, grid, H):
        self.s = s
        self.n, self.K, self.order, self.H = n, grid, s.pme_order, torch.tensor(H, device="cuda")
        self.q, self.radius, self.alpha = _tile(Q, n), _tile(RADIUS, n), _tile(ALPHA, n)
        self.rmin, self.seps, self.mass = _tile(RMIN_HALF, n), _tile(SQRT_EPS, n), _tile(MASS, n)
        self.beta, self.rc_e = s.ewald_beta, s.elec_cutoff if s.split_rows else s.cutoff
        self.self_d = 4 * self.beta**3 / (3 * math.sqrt(math.pi))
        first = 3 * torch.arange(n // 3, device="cuda")
        self.cov = [(first + i, first + j, c) for i, j, c in COV]
        self.mod = []
        th = self._splines(torch.zeros(1, dtype=torch.float64, device="cuda"))[0][0]
        for k in grid:
            arg = 2 * math.pi / k * torch.arange(k, dtype=torch.float64, device="cuda")[:, None] * torch.arange(self.order, dtype=torch.float64, device="cuda")
            b = (th * torch.cos(arg)).sum(1) ** 2 + (th * torch.sin(arg)).sum(1) ** 2
            self.mod.append(torch.where(b < 1e-7, 0.5 * (b.roll(1) + b.roll(-1)), b))

    def _splines(self, f):
        """theta_k = M_P(f + P - 1 - k) and its derivative, (N, P) each."""
        w, prev = [1 - f, f], None
        for n in range(3, self.order + 1):
            prev = w
            # M_n(u) = [u M_(n-1)(u) + (n - u) M_(n-1)(u - 1)] / (n - 1) at u = f + n - 1 - k
            get = lambda k: prev[k] if 0 <= k < len(prev) else torch.zeros_like(f)  # noqa: E731, B023
            w = [((f + n - 1 - k) * get(k - 1) + (1 - f + k) * get(k)) / (n - 1) for k in range(n)]
        get = lambda k: prev[k] if 0 <= k < len(prev) else torch.zeros_like(f)  # noqa: E731
        return torch.stack(w, 1), torch.stack([get(k - 1) - get(k) for k in range(self.order)], 1)

    def perm(self, pos, H):
        p = torch.zeros_like(pos)
        for i, j, c in self.cov:
            v = pos[j] - pos[i]
            v = v - (v - _images(v, H)).detach()
            p = p.index_add(0, i, c * v / v.norm(dim=1, keepdim=True))
        return p

    def _mesh(self, pos, H):
        u = pos @ torch.linalg.inv(H)
        u = (u - torch.floor(u).detach()) * torch.tensor(self.K, device="cuda")
        b = torch.floor(u.detach())
        ax = [self._splines(u[:, a] - b[:, a]) for a in range(3)]
        k = [(b[:, a, None].long() + torch.arange(self.order, device="cuda")) % self.K[a] for a in range(3)]
        at = (k[0][:, :, None, None] * self.K[1] + k[1][:, None, :, None]) * self.K[2] + k[2][:, None, None, :]
        return ax, at

    def _influence(self, H):
        Hinv = torch.linalg.inv(H)
        m = [torch.fft.fftfreq(k, 1 / k, dtype=torch.float64, device="cuda") for k in self.K]
        m[2] = torch.arange(self.K[2] // 2 + 1, dtype=torch.float64, device="cuda")
        v = [m[0][:, None, None] * Hinv[c, 0] + m[1][None, :, None] * Hinv[c, 1] + m[2] * Hinv[c, 2] for c in range(3)]
        m2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
        zero = torch.zeros_like(m2, dtype=torch.bool)
        zero[0, 0, 0] = True
        m2 = torch.where(zero, torch.ones_like(m2), m2)
        g = torch.exp(-math.pi**2 * m2 / self.beta**2) / (2 * math.pi * torch.linalg.det(H).abs() * m2)
        g = g / (self.mod[0][:, None, None] * self.mod[1][None, :, None] * self.mod[2][: self.K[2] // 2 + 1])
        return torch.where(zero, torch.zeros_like(g), g)

    def _spread(self, ax, at, q, d, H):
        e = d @ torch.linalg.inv(H) * torch.tensor(self.K, device="cuda")
        (t1, u1), (t2, u2), (t3, u3) = ax
        c = lambda x, y, z: x[:, :, None, None] * y[:, None, :, None] * z[:, None, None, :]  # noqa: E731
        v = c(q[:, None] * t1 + e[:, :1] * u1, t2, t3) + c(e[:, 1:2] * t1, u2, t3) + c(e[:, 2:] * t1, t2, u3)
        return torch.zeros(math.prod(self.K), dtype=torch.float64, device="cuda").index_add(0, at.flatten(), v.flatten()).view(*self.K)

    def set_geometry(self, pos):
        self.pos = pos
        self.i, self.j = _pair_list(pos, self.H, self.s.cutoff)
        d = pos[self.i] - pos[self.j]
        x = _images(d, self.H)
        self.shift = torch.round((d - x) @ torch.linalg.inv(self.H))
        r = x.norm(dim=1)
        near = r < self.rc_e
        self.ei, self.ej, self.eshift, self.x = self.i[near], self.j[near], self.shift[near], x[near]
        a = torch.rsqrt(2 * (self.radius[self.ei] ** 2 + self.radius[self.ej] ** 2))
        A, B = _screened(a, r[near]), _screened(self.beta, r[near])
        self.g1, self.g2 = (A[1] - B[1])[:, None], (A[2] - B[2])[:, None]
        self.p = self.perm(pos, self.H)
        self.ax, self.at = self._mesh(pos, self.H)
        self.G = self._influence(self.H)

    def gradient(self, q, d):
        """dU/dd of the charges q and dipoles d, in e / nm^2."""
        i, j, x = self.ei, self.ej, self.x
        t = lambda v: self.g1 * v - self.g2 * (v * x).sum(1, keepdim=True) * x  # noqa: E731
        s = torch.zeros_like(d).index_add(0, i, t(d[j]) - self.g1 * q[j, None] * x).index_add(0, j, t(d[i]) + self.g1 * q[i, None] * x)
        F = torch.fft.rfftn(self._spread(self.ax, self.at, q, d, self.H))
        phi = 2 * math.prod(self.K) * torch.fft.irfftn(self.G * F, s=self.K)
        phi = phi.flatten()[self.at]
        (t1, u1), (t2, u2), (t3, u3) = self.ax
        g = [torch.einsum("nijk,ni,nj,nk->n", phi, *w) for w in ((u1, t2, t3), (t1, u2, t3), (t1, t2, u3))]
        return s + torch.stack(g, 1) * torch.tensor(self.K, device="cuda") @ torch.linalg.inv(self.H).T - self.self_d * d

    def solve(self, start=None):
        """The converged induced dipoles."""
        al = self.alpha[:, None]
        zero = torch.zeros_like(self.q)
        b = -self.gradient(self.q, self.p)
        norm = (al * b).abs().mean()
        mul = lambda v: v / al + self.gradient(zero, v)  # noqa: E731
        x = al * b if start is None else start
        r = b - mul(x)
        p = z = al * r
        for _ in range(80):
            rz = (r * z).sum()
            ap = mul(p)
            a = rz / (p * ap).sum()
            x, r = x + a * p, r - a * ap
            z = al * r
            if z.abs().max() < 1e-12 * norm:
                break
            p = z + (r * z).sum() / rz * p
        return x

    def energy(self, mu):
        """(forces, virial, E_elec, E_vdw) at the dipoles mu; the virial is dE/d(strain) with molecular scaling."""
        pos = self.pos.clone().requires_grad_()
        eps = torch.zeros(3, 3, dtype=torch.float64, device="cuda", requires_grad=True)
        y = self.pos.view(-1, 3, 3)
        y = y[:, :1] + _images(y - y[:, :1], self.H)
        com = ((y * self.mass.view(-1, 3, 1)).sum(1) / sum(MASS)).repeat_interleave(3, 0)
        com = com + (self.pos - y.reshape(-1, 3))  # of the atom's own image
        E = torch.zeros(2, dtype=torch.float64, device="cuda")
        scaled = lambda: (pos + com @ eps.T, self.H + self.H @ eps.T)  # noqa: E731
        d_leaf = (mu + self.p).detach().requires_grad_()
        for a in range(0, len(self.ei), 2000000):
            c = slice(a, a + 2000000)
            x_all, H = scaled()
            i, j = self.ei[c], self.ej[c]
            x = x_all[i] - x_all[j] - self.eshift[c] @ H
            al = torch.rsqrt(2 * (self.radius[i] ** 2 + self.radius[j] ** 2))
            r = x.norm(dim=1)
            g0, g1, g2 = (u - v for u, v in zip(_screened(al, r), _screened(self.beta, r)))
            di, dj, qi, qj = d_leaf[i], d_leaf[j], self.q[i], self.q[j]
            dix, djx = (di * x).sum(1), (dj * x).sum(1)
            e = KE * (qi * qj * g0 + (qi * djx - qj * dix) * g1 - g2 * dix * djx + g1 * (di * dj).sum(1)).sum()
            e.backward()
            E[0] += e.detach()
        lj = (self.seps[self.i] * self.seps[self.j] != 0) & (self.i // 3 != self.j // 3)
        i, j, shift = self.i[lj], self.j[lj], self.shift[lj]
        x_all, H = scaled()
        s6 = ((self.rmin[i] + self.rmin[j]) ** 2 / ((x_all[i] - x_all[j] - shift @ H) ** 2).sum(1)) ** 3
        e = (self.seps[i] * self.seps[j] * (s6 * s6 - 2 * s6)).sum()
        e.backward()
        tail = sum(math.comb(6, k) * (self.seps * self.rmin**k).sum() * (self.seps * self.rmin ** (6 - k)).sum() for k in range(7))
        tail = -4 * math.pi * tail / (3 * torch.linalg.det(self.H).abs() * self.s.cutoff**3)
        E[1] = e.detach() + tail
        x_all, H = scaled()
        ax, at = self._mesh(x_all, H)
        F = torch.fft.rfftn(self._spread(ax, at, self.q, d_leaf, H))
        w = torch.full((self.K[2] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = w[-1] = 1.0
        e = KE * ((w * self._influence(H) * (F.real**2 + F.imag**2)).sum() - self.beta / math.sqrt(math.pi) * (self.q**2).sum()
                  - 0.5 * self.self_d * (d_leaf**2).sum() + (mu * mu / (2 * self.alpha[:, None])).sum())
        e.backward()
        E[0] += e.detach()
        self.perm(pos, self.H).backward(d_leaf.grad)  # the molecules are rigid under the strain: so are their dipoles
        return -pos.grad, eps.grad - 2 * tail * torch.eye(3, dtype=torch.float64, device="cuda"), E[0], E[1]


def _mesh_size(H, spacing):
    """The smallest even mesh of factors 2, 3, 5 with planes at most `spacing` apart."""
    smooth = [k for k in range(8, 257, 2) if 2**8 * 3**5 * 5**3 % k == 0]
    heights = [abs(np.linalg.det(H)) / np.linalg.norm(np.cross(H[a - 2], H[a - 1])) for a in range(3)]
    return tuple(next(k for k in smooth if k >= math.ceil(h / spacing)) for h in heights)


def _models(case, pos, boxes):
    s = _settings(case)
    return [_Model(len(x), s, tuple(s.pme_grid) if s.pme_grid else _mesh_size(H, s.pme_spacing), H) for x, H in zip(pos, boxes)]


def _forces(models, xs, mus):
    out = []
    for k, (m, x) in enumerate(zip(models, xs)):
        m.set_geometry(x)
        mus[k] = m.solve(mus[k])
        out.append(m.energy(mus[k])[0])
    return out


def _turn(k, t, inertia, L, R):
    """Free rotation about body axis k for a time t (L in the body frame, R body -> space)."""
    phi = t * L[:, k] / inertia[k]
    c, s = torch.cos(phi), torch.sin(phi)
    a, b = (k + 1) % 3, (k + 2) % 3
    L, R = L.clone(), R.clone()
    L[:, a], L[:, b] = c * L[:, a] + s * L[:, b], c * L[:, b] - s * L[:, a]
    R[:, :, a], R[:, :, b] = c[:, None] * R[:, :, a] + s[:, None] * R[:, :, b], c[:, None] * R[:, :, b] - s[:, None] * R[:, :, a]
    return L, R


def _md_values(case, seed):
    """WARM + 1 velocity-Verlet steps of the rigid molecules."""
    pos, vel, boxes = _inputs(case, seed)
    models, sizes = _models(case, pos, boxes), [len(x) for x in pos]
    m = torch.tensor(MASS, dtype=torch.float64, device="cuda")
    x, v = (torch.from_numpy(np.concatenate(a)).cuda().view(-1, 3, 3) for a in (pos, vel))
    edge = torch.cat([torch.full((n // 3, 1), H[0, 0], dtype=torch.float64, device="cuda") for n, H in zip(sizes, boxes)])
    com = (m[:, None] * x).sum(1) / m.sum()
    y = x - com[:, None]
    inertia = (m[:, None, None] * ((y[0] ** 2).sum(1)[:, None, None] * torch.eye(3, device="cuda") - y[0][:, :, None] * y[0][:, None])).sum(0)
    inertia, axes = torch.linalg.eigh(inertia)
    axes[:, 0] *= torch.linalg.det(axes).sign()
    body = y[0] @ axes
    U, _, Vt = torch.linalg.svd(body.T @ y)
    flip = torch.diag_embed(torch.stack([torch.ones_like(edge[:, 0])] * 2 + [torch.linalg.det(U @ Vt).sign()], 1))
    R = Vt.transpose(1, 2) @ flip @ U.transpose(1, 2)
    P = (m[:, None] * v).sum(1)
    L = (R.transpose(1, 2) @ (m[:, None] * torch.linalg.cross((R @ body.T).transpose(1, 2), v)).sum(1)[:, :, None])[:, :, 0]
    mus = [None] * len(models)

    def kick(F, P, L):
        F = torch.cat(F).view(-1, 3, 3)
        torque = torch.linalg.cross((R @ body.T).transpose(1, 2), F).sum(1)
        return P + 0.5 * DT * F.sum(1), L + 0.5 * DT * (R.transpose(1, 2) @ torque[:, :, None])[:, :, 0]

    def positions(com):
        com = com - torch.floor(com / edge) * edge
        return com, (com[:, None] + (R @ body.T).transpose(1, 2)).reshape(-1, 3)

    com, x = positions(com)
    F = _forces(models, x.split(sizes), mus)
    for _ in range(WARM + 1):
        P, L = kick(F, P, L)
        com = com + DT * P / m.sum()
        for axis, h in ((2, 0.5), (1, 0.5), (0, 1.0), (1, 0.5), (2, 0.5)):
            L, R = _turn(axis, h * DT, inertia, L, R)
        com, x = positions(com)
        F = _forces(models, x.split(sizes), mus)
        P, L = kick(F, P, L)
    return {"pos": x, "mom": P, "forces": torch.cat(F), "mu": torch.cat(mus)}


def _bonded(q):
    """Forces of the flexible molecules' own surface; q (beads n, 3)."""
    D, al, r0, kth, th0 = BOND
    x = q.detach().clone().requires_grad_()
    m = x.view(-1, 3, 3)
    u, v = m[:, 1] - m[:, 0], m[:, 2] - m[:, 0]
    e = sum(D * (a**2 - a**3 + 7 / 12 * a**4) for a in (al * (u.norm(dim=1) - r0), al * (v.norm(dim=1) - r0)))
    th = torch.acos((u * v).sum(1) / (u.norm(dim=1) * v.norm(dim=1)))
    (e + 0.5 * kth * (th - th0) ** 2).sum().backward()
    return -x.grad


def _pimd_values(case, seed):
    """WARM + 1 steps of ring-polymer MD: kick, free ring polymer, kick."""
    (pos,), _, (H,) = _inputs(case, seed)
    P, n, h = case["systems"], len(pos), DT / 2
    kT = P * KB * 300.0
    mass = np.tile(MASS, n // 3)
    j, l = np.arange(P)[:, None], (np.arange(P) + 1) // 2
    C = np.where(np.arange(P) % 2 == 1, np.cos(2 * np.pi * j * l / P), np.sin(2 * np.pi * j * l / P)) * math.sqrt(2 / P)
    C[:, 0] = 1 / math.sqrt(P)
    if P % 2 == 0:
        C[:, -1] = (-1.0) ** j[:, 0] / math.sqrt(P)
    om = 2 * kT / HBAR * np.sin(np.pi * l / P)
    rng = np.random.default_rng(seed)
    y = np.zeros((P, n, 3))
    y[0] = math.sqrt(P) * pos
    for k in range(1, P):
        y[k] = rng.normal(size=(n, 3)) * np.sqrt(kT / mass)[:, None] / om[k]
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    C, w, m = t(C), t(om)[:, None, None], t(mass)[None, :, None]
    p = t(rng.normal(size=(P, n, 3))) * torch.sqrt(kT * m)
    q = torch.einsum("jl,lnc->jnc", C, t(y))
    models, mus = _models(case, [pos] * P, [H] * P), [None] * P
    force = lambda q: (torch.cat(_forces(models, list(q), mus)) + _bonded(q.reshape(-1, 3))).view(P, n, 3)  # noqa: E731
    F = force(q)
    for _ in range(WARM + 1):
        p = p + 0.5 * h * F
        qn, pn = torch.einsum("jl,jnc->lnc", C, q), torch.einsum("jl,jnc->lnc", C, p)
        for _half in range(2):
            s, z = 0.5 * h, 0.25 * (w * 0.5 * h) ** 2
            qn, pn = (s * pn / m + (1 - z) * qn) / (1 + z), ((1 - z) * pn - m * w * w * s * qn) / (1 + z)
        q, p = torch.einsum("jl,lnc->jnc", C, qn), torch.einsum("jl,lnc->jnc", C, pn)
        F = force(q)
        p = p + 0.5 * h * F
    return {"pos": q.reshape(-1, 3), "mom": p.reshape(-1, 3), "forces": F.reshape(-1, 3), "mu": torch.cat(mus)}


def _train_values(case, seed):
    """Loss, weights and moments after one Adam step (learning rate 1e-3)."""
    f, w = _train_inputs(case, seed)
    w = w.double().requires_grad_()
    W = [p.view(*s) for p, s in zip(w.split([math.prod(s) for s in MPNN_SHAPES]), MPNN_SHAPES)]
    n, silu = len(f["inv"]), torch.nn.functional.silu
    i = torch.arange(n, device="cuda").repeat_interleave(f["counts"].long())
    e = f["edges"][torch.arange(EMAX, device="cuda") < f["counts"][:, None]]
    j = e[:, 3].contiguous().view(torch.int32).long()
    d = e[:, :3].double().norm(dim=1, keepdim=True)
    c = torch.arange(8, dtype=torch.float64, device="cuda") * (GRAPH_CUTOFF / 7)
    phi = torch.exp(-((7 / GRAPH_CUTOFF * (d - c)) ** 2)) * 0.5 * (torch.cos(math.pi * d / GRAPH_CUTOFF) + 1)
    h = silu(f["inv"].double() @ W[0].T + W[1])
    for k in (2, 8):
        Wg, Wf, Wa, ba, Wb, bb = W[k:k + 6]
        a = torch.zeros(n, 16, dtype=torch.float64, device="cuda").index_add(0, i, (phi @ Wf.T) * (h @ Wg.T)[j])
        h = h + silu(torch.cat([h, a], 1) @ Wa.T + ba) @ Wb.T + bb
    mu = SIGMA * torch.einsum("nc,nck->nk", (h @ W[-2].T + W[-1])[:, :15], f["vec"].double())
    loss = ((mu - f["target"].double()) ** 2).sum() / (n * SIGMA**2)
    loss.backward()
    g = w.grad
    return {"loss": float(loss), "w": (w - 1e-3 * g / (g.abs() + 1e-8)).detach(), "m": 0.1 * g, "v": 0.001 * g * g}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_values(case, seed)
    if kind == "md":
        return _md_values(case, seed)
    if kind == "pimd":
        return _pimd_values(case, seed)
    (pos,), _, (H,) = _inputs(case, seed)
    if kind == "host":
        pos = _trajectory(pos, seed)[WARM]
    (m,) = _models(case, [pos], [H])
    m.set_geometry(torch.from_numpy(np.ascontiguousarray(pos)).cuda())
    if kind == "field":
        return -m.gradient(m.q, torch.from_numpy(_dipoles(m.n, seed)).cuda())
    mu = m.solve()
    forces, virial, elec, vdw = m.energy(mu)
    if kind == "host":
        return {"forces": forces}
    out = {"forces": forces, "mu": mu}
    if case["precision"] == "double":
        out.update(energy=(elec + vdw).view(1), elec=elec.view(1), vdw=vdw.view(1), virial=virial[None])
    return out
