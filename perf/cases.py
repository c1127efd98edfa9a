"""The work that a user of this framework has it do, as cases that can be timed
and compared: each goes through the public entry points (openpixi_gb300.Handle and
Batch, the ctypes form of include/opixi.h) and returns what the path computes.

A case is one of six kinds:

  run       a pure Yang-Mills simulation: `steps` leapfrog steps, the
            BulkQuantities row of every step (measured) or of the last one, and a
            snapshot of the new links and electric fields into page-locked memory
  batch     many independent lattices advanced together, their BulkQuantities
            rows and a snapshot of each
  collision the CPIC loop: fields and NGP particles, the BulkQuantities and
            ProjectedEnergyDensity rows of every step, the fields at the end
  gradient  the adjoint of the mean energy density with respect to the initial E
  drop_in   FieldSolver.step for a host program that keeps its grid in its own
            (pageable) memory: U and E in, one update, E and Unext out
  project   RandomGaussianFields: the projection of E onto Gauss's law

Inputs are Gaussian links U = exp(i A^a t_a) and fields E of the widths that the
benchmark and the input decks use, drawn with torch on the GPU from the seed.
Fields of an FP32 handle are returned as float32 (the device's type), so are its
rows; the C ABI hands every value over as a double.
"""
import math

import numpy as np
import torch

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

DEV = "cuda"
EVENT_SIZES = (16, 24, 32, 40, 48)  # the batching workload's lattice sizes


def listed():
    return [
        # the headline workload of bench.py with BulkQuantitiesInTime at every step
        # (MainBatch's loop), 100 of its steps
        dict(name="su3_f32_128_measured", kind="run", nc=3, prec="f32", n0=128, n1=128, n2=128, steps=100, sigma=0.2,
             measured=True),
        # a lattice whose sizes are no multiples of anything, diagnostics at the end
        dict(name="su3_f32_ragged", kind="run", nc=3, prec="f32", n0=50, n1=45, n2=70, steps=100, sigma=0.2,
             measured=False),
        # the SU(2) FP32 workload of the lattice-size sweep
        dict(name="su2_f32_128", kind="run", nc=2, prec="f32", n0=128, n1=128, n2=128, steps=100, sigma=0.1,
             measured=False),
        # the plain FP64 parity workload (32^3, dt = 0.05, 100 steps), measured
        dict(name="su2_f64_32", kind="run", nc=2, prec="f64", n0=32, n1=32, n2=32, steps=100, sigma=0.1, measured=True),
        # the plain FP64 form of SU(3)
        dict(name="su3_f64_40", kind="run", nc=3, prec="f64", n0=40, n1=40, n2=40, steps=10, sigma=0.2, measured=True),
        # an ensemble of SU(2) events of uneven sizes, 200 steps (the batching workload, a quarter of its events)
        dict(name="batch_su2", kind="batch", nc=2, events=64, steps=200, sigma=0.1),
        # the same for SU(3)
        dict(name="batch_su3", kind="batch", nc=3, events=32, steps=50, sigma=0.1),
        # the CPIC collision lattice with two beams of two particles a cell, diagnostics every step
        dict(name="collision", kind="collision", n0=256, n1=64, n2=64, steps=8, sigma=0.05),
        # the differentiation workload's lattice, a part of its 200 steps between checkpoints every 14
        dict(name="gradient_64", kind="gradient", n=64, steps=42, ckpt=14, sigma=0.1),
        # a small per-call drop-in: latency
        dict(name="drop_in_16", kind="drop_in", nc=2, n0=16, n1=16, n2=16, sigma=0.1),
        # the initial condition of an SU(3) FP32 run
        dict(name="project_su3_64", kind="project", nc=3, prec="f32", n0=64, n1=64, n2=64, sigma=0.2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, vmin, vmax):
    """Three sides whose product is about a log-uniform volume, of uneven shape."""
    v = _log(rng, vmin, vmax)
    f = [_log(rng, 0.6, 1.7) for _ in range(3)]
    s = (v / (f[0] * f[1] * f[2])) ** (1.0 / 3.0)
    d = [max(2, int(round(s * x))) for x in f]
    while d[0] * d[1] * d[2] > vmax:
        d[d.index(max(d))] -= 1
    return dict(n0=d[0], n1=d[1], n2=d[2])


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "batch", "collision", "gradient", "drop_in", "project"])
    nc = rng.choice([2, 3])
    sigma = round(rng.uniform(0.08, 0.22), 3)
    if kind == "run":
        prec = rng.choice(["f32", "f32", "f64"])
        vmax = 128 ** 3 if prec == "f32" else (64 ** 3 if nc == 2 else 40 ** 3)
        steps = rng.randint(20, 100) if prec == "f32" or nc == 2 else rng.randint(3, 10)
        return dict(kind=kind, nc=nc, prec=prec, steps=steps, sigma=sigma, measured=rng.random() < 0.5,
                    **_dims(rng, 10 ** 3, vmax))
    if kind == "batch":
        return dict(kind=kind, nc=nc, events=int(_log(rng, 3, 65 if nc == 2 else 33)), steps=rng.randint(20, 50),
                    sigma=min(sigma, 0.15))
    if kind == "collision":
        n0, n1, n2 = rng.randint(32, 256), rng.randint(8, 64), rng.randint(8, 64)
        return dict(kind=kind, n0=n0, n1=n1, n2=n2, steps=rng.randint(2, 8), sigma=0.05)
    if kind == "gradient":
        return dict(kind=kind, n=int(_log(rng, 8, 64.99)), steps=rng.randint(5, 42), ckpt=rng.randint(3, 14),
                    sigma=min(sigma, 0.12))
    if kind == "drop_in":
        return dict(kind=kind, nc=nc, sigma=sigma, **_dims(rng, 5 ** 3, 32 ** 3))
    prec = rng.choice(["f32", "f64"])
    return dict(kind=kind, nc=nc, prec=prec, sigma=sigma, **_dims(rng, 8 ** 3, 64 ** 3))


# ------------------------------------------------------------------ inputs
def _lambdas(nc):
    """Generators t_a = lambda_a / 2 as complex matrices [na, nc, nc]."""
    if nc == 2:
        m = [[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]]
    else:
        r = 1 / math.sqrt(3.0)
        m = [[[0, 1, 0], [1, 0, 0], [0, 0, 0]], [[0, -1j, 0], [1j, 0, 0], [0, 0, 0]], [[1, 0, 0], [0, -1, 0], [0, 0, 0]],
             [[0, 0, 1], [0, 0, 0], [1, 0, 0]], [[0, 0, -1j], [0, 0, 0], [1j, 0, 0]], [[0, 0, 0], [0, 0, 1], [0, 1, 0]],
             [[0, 0, 0], [0, 0, -1j], [0, 1j, 0]], [[r, 0, 0], [0, r, 0], [0, 0, -2 * r]]]
    return torch.tensor(m, dtype=torch.complex128, device=DEV) / 2


def _mul(a, b):
    """Matrix product of fields [nc, nc, ...]."""
    out = a[:, 0:1] * b[0:1]
    for k in range(1, a.shape[1]):
        out = out + a[:, k:k + 1] * b[k:k + 1]
    return out


def _adj(a):
    return a.transpose(0, 1).conj()


def _herm(x, t):
    """x^a t_a for generator components x [na, ...] (real)."""
    return torch.tensordot(t.permute(1, 2, 0), x.to(torch.complex128), dims=1)


def _expi(h, order):
    """exp(i h) of a hermitian field by its Taylor polynomial (Horner)."""
    one = torch.eye(h.shape[0], dtype=torch.complex128, device=DEV).reshape(h.shape[:2] + (1,) * (h.dim() - 2))
    out = one + 1j * h / order
    for k in range(order - 1, 0, -1):
        out = one + _mul(1j * h / k, out)
    return out


def _fields(nc, shape, sigma, seed):
    """U: three link fields [nc, nc, *shape] and E: three of generator components [na, *shape]."""
    t = _lambdas(nc)
    g = torch.Generator(device=DEV).manual_seed(seed)
    U, E = [], []
    for _ in range(3):
        a = torch.randn((t.shape[0],) + shape, generator=g, device=DEV, dtype=torch.float64) * sigma
        U.append(_expi(_herm(a, t), 22))
        E.append(torch.randn((t.shape[0],) + shape, generator=g, device=DEV, dtype=torch.float64) * sigma)
    return U, E


def _links_ref(U):
    """Three link fields to the ABI's layout [V][3][4 or 18] (on the GPU)."""
    rows = []
    for u in U:
        u = u.reshape(u.shape[0], u.shape[1], -1)
        if u.shape[0] == 2:  # e0 + i e_a sigma_a
            rows.append(torch.stack([u[0, 0].real, u[0, 1].imag, u[0, 1].real, u[0, 0].imag]))
        else:
            m = u.reshape(9, -1)
            rows.append(torch.cat([m.real, m.imag]))
    return torch.stack(rows).permute(2, 0, 1).contiguous()


def _alg_gen(E):
    """Three fields of generator components to [V][3][na]."""
    return torch.stack([e.reshape(e.shape[0], -1) for e in E]).permute(2, 0, 1).contiguous()


def _prec(case):
    return opx.OPX_F32 if case.get("prec") == "f32" else opx.OPX_F64


def _event_dims(case):
    return [EVENT_SIZES[(7 * q * q + 3 * q + q // 5) % 5] for q in range(case["events"])]


class _Snapshot:
    """Page-locked doubles that a download writes, and the float32 copy that an FP32 run keeps."""

    def __init__(self, shape, f32):
        self.pinned = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        self.doubles = self.pinned.numpy()
        self.single = torch.empty(shape, dtype=torch.float32) if f32 else None

    def result(self):
        return self.pinned if self.single is None else self.single.copy_(self.pinned)


def _rows(obs, f32=False):
    r = np.array([list(o.e2) + list(o.b2) + [o.px, o.py, o.pz, o.gauss, o.rho2, o.e2_total, o.b2_total] for o in obs])
    return r.astype(np.float32) if f32 else r


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        nc, sizes = case["nc"], _event_dims(case)
        b = opx.Batch(nc, [(L, L, L) for L in sizes], dt=0.05, precision=opx.OPX_F32, reunit_every=10)
        for L in sorted(set(sizes)):
            at = [q for q, M in enumerate(sizes) if M == L]
            U, E = _fields(nc, (len(at), L, L, L), case["sigma"], seed + L)
            for k, q in enumerate(at):
                b.upload(q, opx.FIELD_U, _links_ref([u[:, :, k] for u in U]).cpu().numpy())
                b.upload(q, opx.FIELD_E, _alg_gen([e[:, k] for e in E]).cpu().numpy(), layout=opx.LAYOUT_GEN)
        b.initialize()
        b.autotune(steps=3)
        V = sum(L ** 3 for L in sizes)
        return dict(case=case, b=b, sizes=sizes, links=_Snapshot((V, 3, b.ng), True), e=_Snapshot((V, 3, b.ngen), True))
    dims = (case["n"],) * 3 if kind == "gradient" else (case["n0"], case["n1"], case["n2"])
    nc = 2 if kind in ("gradient", "collision") else case["nc"]
    f32 = case.get("prec") == "f32"
    dt = 0.5 if kind == "collision" else 0.05
    h = opx.Handle(nc, dims, a=1.0, dt=dt, g=1.0, precision=_prec(case), reunit_every=10 if f32 else 0)
    U, E = _fields(nc, dims, case["sigma"], seed)
    U, E = _links_ref(U).cpu().numpy(), _alg_gen(E).cpu().numpy()
    if kind == "drop_in":
        return dict(case=case, h=h, U=U, E=E, Unext=np.empty_like(U), Enew=np.empty_like(E))
    h.upload(opx.FIELD_U, U)
    h.upload(opx.FIELD_E, E, layout=opx.LAYOUT_GEN)
    if kind == "project":
        return dict(case=case, h=h, E=torch.from_numpy(E).pin_memory(), e=_Snapshot(E.shape, f32))
    if kind == "gradient":
        return dict(case=case, h=h)
    if kind == "collision":
        h.particles_upload(*_particles(case, seed))
    h.initialize()
    return dict(case=case, h=h, links=_Snapshot(U.shape, f32), e=_Snapshot(E.shape, f32))


def _particles(case, seed):
    """Two beams along direction 0, each over a quarter of the lattice: two particles in a cell."""
    n0, n1, n2 = case["n0"], case["n1"], case["n2"]
    pos, vel = [], []
    for first, v in ((n0 // 8, 1.0), (n0 - n0 // 8 - n0 // 4, -1.0)):
        x = np.stack(np.meshgrid(np.arange(first, first + n0 // 4), np.arange(n1), np.arange(n2), [-0.25, 0.25],
                                 indexing="ij"), -1).reshape(-1, 4)
        pos.append(np.stack([x[:, 0] + x[:, 3], x[:, 1], x[:, 2]], -1))
        vel.append(np.tile([v, 0.0, 0.0], (len(x), 1)))
    pos, vel = np.concatenate(pos), np.concatenate(vel)
    q = np.random.default_rng(seed).normal(0.0, 0.05, (len(pos), 3))
    return pos, pos - 0.5 * vel, vel, q, q.copy(), np.zeros(len(pos), np.int32)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "batch":
        b, o = state["b"], 0
        b.run(case["steps"])
        rows = _rows(b.reduce(), True)
        for q, L in enumerate(state["sizes"]):
            V = L ** 3
            for field, layout, to in ((opx.FIELD_UNEXT, opx.LAYOUT_REF, state["links"]), (opx.FIELD_E, opx.LAYOUT_GEN, state["e"])):
                part = to.doubles[o:o + V]
                b.check(b.L.opx_batch_download(b.h, q, field, N.ptr(part), part.size, layout))
            o += V
        return dict(rows=rows, links=state["links"].result(), e=state["e"].result())
    h = state["h"]
    f32 = case.get("prec") == "f32"
    if kind == "drop_in":
        h.upload(opx.FIELD_U, state["U"])
        h.upload(opx.FIELD_E, state["E"], layout=opx.LAYOUT_GEN)
        h.update_grid()
        return dict(e=h.download(opx.FIELD_E, layout=opx.LAYOUT_GEN, out=state["Enew"]),
                    links=h.download(opx.FIELD_UNEXT, out=state["Unext"]))
    if kind == "project":
        h.upload(opx.FIELD_E, state["E"].numpy(), layout=opx.LAYOUT_GEN)
        h.gauss_project(1e-26)
        h.download(opx.FIELD_E, layout=opx.LAYOUT_GEN, out=state["e"].doubles)
        return dict(e=state["e"].result())
    if kind == "gradient":
        lo, hi = _box(case)
        J, g = h.energy_gradient(case["steps"], case["ckpt"], lo, hi)
        return dict(J=J, gradient=g)
    out = {}
    if kind == "collision":
        rows, slices = [], []
        for _ in range(case["steps"]):
            h.step(1)
            rows.append(h.reduce())
            slices.append(h.projected_energy(0))
        out["slices"] = np.stack(slices)
    elif case["measured"]:
        rows = h.step_measured(case["steps"])
    else:
        h.step(case["steps"])
        rows = [h.reduce()]
    out["rows"] = _rows(rows, f32)
    h.download(opx.FIELD_UNEXT, out=state["links"].doubles)
    out["links"] = state["links"].result()
    h.download(opx.FIELD_E, layout=opx.LAYOUT_GEN, out=state["e"].doubles)
    out["e"] = state["e"].result()
    return out


def _box(case):
    n = case["n"]
    return (n // 2 - n // 8,) * 3, (n // 2 + n // 8 - 1,) * 3


# ------------------------------------------------------------------ work
# Per link update: bytes of U and E read and of E and Unext written (FP32), and
# operations of the plaquette form (a plaquette's three products shared by its
# four links, each transport once, one exponential and one product with it),
# an FMA counted as two.
LINK_BYTES = {2: 56, 3: 208}
LINK_FLOPS = {2: 260, 3: 1800}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        V, nc, r, n = sum(L ** 3 for L in _event_dims(case)), case["nc"], 1, case["steps"]
    else:
        V = case["n"] ** 3 if kind == "gradient" else case["n0"] * case["n1"] * case["n2"]
        nc = 2 if kind in ("gradient", "collision") else case["nc"]
        r = 1 if case.get("prec") == "f32" else 2
        n = case.get("steps", 1)
    ng, na = (4, 3) if nc == 2 else (18, 8)
    snapshot = V * 3 * (ng + na) * (4 * r + 8)  # device values read, doubles written
    step_b, step_f = 3 * V * LINK_BYTES[nc] * r, 3 * V * LINK_FLOPS[nc]
    if kind == "project":
        # links, the charge and E once, E written; of the order of 100 Laplacians of six transports
        return {"bytes": V * 4 * r * (3 * ng + 7 * na) + 16 * V * 3 * na, "flops": 100.0 * V * 6 * (36 if nc == 2 else 320)}
    if kind == "gradient":
        # forward once, its states kept, and the reverse of every step (about twice a step's work)
        return {"bytes": n * 3 * step_b + 8 * V * 9, "flops": n * 3 * step_f}
    if kind == "drop_in":
        return {"bytes": step_b + 2 * snapshot, "flops": step_f}
    if kind == "collision":
        p = 4 * (case["n0"] // 4) * case["n1"] * case["n2"]
        return {"bytes": n * (step_b + V * (96 + 96 + 24) + p * 209) + snapshot, "flops": n * (step_f + p * 60 + V * 300)}
    return {"bytes": n * step_b + snapshot, "flops": n * step_f * (1.25 if case.get("measured") else 1)}


# ------------------------------------------------------------------ the same in 64 bits with plain torch
def _roll(x, d, o):
    """The field at y + o d as seen from y (three trailing lattice dimensions)."""
    return torch.roll(x, -o, dims=x.dim() - 3 + d)


def _proj(m, t):
    """Im tr(lambda_a m), lambda = 2 t."""
    return 2 * torch.einsum("aij,ji...->a...", t, m).imag


def _force(U, i, t):
    S = 0
    for j in range(3):
        if j == i:
            continue
        S = S + _mul(_mul(_roll(U[j], i, 1), _adj(_roll(U[i], j, 1))), _adj(U[j]))
        Uj = _roll(U[j], j, -1)
        S = S + _mul(_adj(_mul(_roll(U[i], j, -1), _roll(Uj, i, 1))), Uj)
    return _proj(_mul(U[i], S), t)


def _links_step(U, E, dt, t):
    return [_mul(_expi(_herm(-dt * E[i], t), 14), U[i]) for i in range(3)]


def _step(U, E, dt, t, J=None):
    """One update (a = g = 1) of the new links U: the new E and the next links."""
    E = [E[i] + dt * _force(U, i, t) - (0 if J is None else dt * J[i]) for i in range(3)]
    return E, _links_step(U, E, dt, t)


def _plaquette(U, j, k):
    return _mul(_mul(_mul(U[j], _roll(U[k], j, 1)), _adj(_roll(U[j], k, 1))), _adj(U[k]))


def _square(x):
    return (x * x).sum(0)


def _observables(U, Un, E, t, rho=None):
    """The BulkQuantities row, over the last three dimensions: [..., 13]."""
    V = U[0].shape[-1] * U[0].shape[-2] * U[0].shape[-3]
    tot = lambda x: x.sum((-3, -2, -1)) / V  # noqa: E731
    e2 = [tot(_square(E[d])) for d in range(3)]
    b2 = [tot(_square(_proj(_plaquette(U, (d + 1) % 3, (d + 2) % 3), t)) +
              _square(_proj(_plaquette(Un, (d + 1) % 3, (d + 2) % 3), t))) / 2 for d in range(3)]
    s = [e + b for e, b in zip(e2, b2)]
    G = _gauss(U, E, t) - (0 if rho is None else rho)
    r2 = torch.zeros_like(e2[0]) if rho is None else torch.sqrt(tot(_square(rho)) * V) / V
    return torch.stack(e2 + b2 + [-s[0] + s[1] + s[2], s[0] - s[1] + s[2], s[0] + s[1] - s[2], tot(_square(G)), r2,
                                  sum(e2), sum(b2)], -1)


def _act(x, u, t):
    """Components of u X u^dagger."""
    return 2 * torch.einsum("aij,ji...->a...", t, _mul(_mul(u, _herm(x, t)), _adj(u))).real


def _gauss(U, E, t):
    return sum(E[i] - _roll(_act(E[i], _adj(U[i]), t), i, -1) for i in range(3))


def _slices(U, Un, E, t):
    """ProjectedEnergyDensity along direction 0: rows T_el, T_mag, L_el, L_mag."""
    n0, n1, n2 = E[0].shape[-3:]
    el = [0.5 * _square(E[d]).sum((-2, -1)) / (n1 * n2) for d in range(3)]
    mag = [0.25 * (_square(_proj(_plaquette(U, (d + 1) % 3, (d + 2) % 3), t)) +
                   _square(_proj(_plaquette(Un, (d + 1) % 3, (d + 2) % 3), t))).sum((-2, -1)) / (n1 * n2) for d in range(3)]
    return torch.stack([el[1] + el[2], mag[1] + mag[2], el[0], mag[0]])


class _Beams:
    """The CPIC phases of one step for particles moving along direction 0 (a = 1)."""

    def __init__(self, case, seed, t):
        pos, _, vel, q, _, _ = _particles(case, seed)
        self.dims, self.t = (case["n0"], case["n1"], case["n2"]), t
        self.x = torch.from_numpy(pos).to(DEV)
        self.v = torch.from_numpy(vel[:, 0].copy()).to(DEV)
        self.q0 = torch.from_numpy(q.T.copy()).to(DEV)

    def cell(self, x0):
        n0, n1, n2 = self.dims
        return (torch.remainder(torch.round(x0).long(), n0) * n1 + self.x[:, 1].long()) * n2 + self.x[:, 2].long()

    def phases(self, Un, dt):
        """rho and J_0 of the particles; they move and their charges with them."""
        old = self.cell(self.x[:, 0])
        flat = lambda v, at: torch.zeros((3, int(np.prod(self.dims))), dtype=torch.float64, device=DEV).index_add_(  # noqa: E731
            1, at, v).reshape((3,) + self.dims)
        rho = flat(self.q0, old)
        x1 = self.x[:, 0] + self.v * dt
        new, right = self.cell(x1), self.v > 0
        moved = torch.round(self.x[:, 0]) != torch.round(x1)
        u = Un[0].reshape(2, 2, -1)[:, :, torch.where(right, old, new)]
        u = torch.where(right, _adj(u), u)
        to = _act(self.q0, u, self.t)
        J = flat(torch.where(moved, torch.where(right, self.q0, -to) / dt, 0.0), torch.where(right, old, new))
        self.x[:, 0] = x1
        # a charge that crossed into the next cell goes on transported
        self.q0 = torch.where(moved, to, self.q0)
        return rho, J


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        t, sizes = _lambdas(case["nc"]), _event_dims(case)
        rows, links, e = [None] * len(sizes), [None] * len(sizes), [None] * len(sizes)
        for L in sorted(set(sizes)):
            at = [q for q, M in enumerate(sizes) if M == L]
            U, E = _fields(case["nc"], (len(at), L, L, L), case["sigma"], seed + L)
            Un = _links_step(U, E, 0.05, t)
            for _ in range(case["steps"]):
                U = Un
                E, Un = _step(U, E, 0.05, t)
            obs = _observables(U, Un, E, t)
            for k, q in enumerate(at):
                rows[q] = obs[k].cpu().numpy()
                links[q] = _links_ref([u[:, :, k] for u in Un]).cpu()
                e[q] = _alg_gen([x[:, k] for x in E]).cpu()
        return dict(rows=np.stack(rows), links=torch.cat(links), e=torch.cat(e))
    dims = (case["n"],) * 3 if kind == "gradient" else (case["n0"], case["n1"], case["n2"])
    nc = 2 if kind in ("gradient", "collision") else case["nc"]
    t = _lambdas(nc)
    U, E = _fields(nc, dims, case["sigma"], seed)
    if kind == "drop_in":
        E, Un = _step(U, E, 0.05, t)
        return dict(e=_alg_gen(E), links=_links_ref(Un))
    if kind == "project":
        return dict(e=_alg_gen(_projected(U, E, t)))
    if kind == "gradient":
        return _gradient(case, U, E, t)
    dt = 0.5 if kind == "collision" else 0.05
    Un = _links_step(U, E, dt, t)
    rho = J = None
    rows, slices = [], []
    if kind == "collision":
        beams = _Beams(case, seed, t)
        rho, J = beams.phases(Un, dt)
    for n in range(case["steps"]):
        U = Un
        E, Un = _step(U, E, dt, t, None if J is None else [J, 0 * J, 0 * J])
        if kind == "collision":
            rho, J = beams.phases(Un, dt)
            slices.append(_slices(U, Un, E, t))
        if kind == "collision" or case["measured"] or n + 1 == case["steps"]:
            rows.append(_observables(U, Un, E, t, rho))
    out = dict(rows=torch.stack(rows), links=_links_ref(Un), e=_alg_gen(E))
    if slices:
        out["slices"] = torch.stack(slices)
    return out


def _projected(U, E, t):
    """E + divT K^+ (-div E) by conjugate gradients."""
    divT = lambda l: [l - _act(_roll(l, i, 1), U[i], t) for i in range(3)]  # noqa: E731
    r = -_gauss(U, E, t)
    p, mu, rr = r, torch.zeros_like(r), (r * r).sum()
    V = r[0].numel()
    for _ in range(3000):
        if rr / V <= 1e-30:
            break
        Ap = _gauss(U, divT(p), t)
        al = rr / (p * Ap).sum()
        mu, r = mu + al * p, r - al * Ap
        new = (r * r).sum()
        p, rr = r + (new / rr) * p, new
    return [e + d for e, d in zip(E, divT(mu))]


def _gradient(case, U, E0, t):
    """J and dJ/dE_0 by automatic differentiation, each step recomputed on the way back."""
    from torch.utils.checkpoint import checkpoint
    lo, hi = _box(case)
    E0 = [e.requires_grad_() for e in E0]

    def step(*a):
        E, Un = _step(a[:3], a[3:], 0.05, t)
        return (*Un, *E)

    Un, E, before = _links_step(U, E0, 0.05, t), E0, None
    for _ in range(case["steps"]):
        before = Un
        r = checkpoint(step, *Un, *E, use_reentrant=False)
        Un, E = list(r[:3]), list(r[3:])
    density = 0
    for d in range(3):
        j, k = (d + 1) % 3, (d + 2) % 3
        density = density + 0.5 * _square(E[d]) + 0.25 * _square(_proj(_plaquette(before, j, k), t) +
                                                                 _proj(_plaquette(Un, j, k), t))
    J = density[tuple(slice(a, b + 1) for a, b in zip(lo, hi))].mean()
    J.backward()
    return dict(J=float(J.detach()), gradient=_alg_gen([e.grad for e in E0]))
