"""The workloads by which this library's speed is followed, and their results in plain 64-bit torch.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a user's program holds before the call (the
plan, the spins on the GPU, the dynamics object), ``run(state)`` makes one call
through the package's public entry points, ``work(case)`` counts the bytes and
operations that the call cannot do without, and ``exact(case, seed)`` restates
the call's result with torch tensor operations alone (neighbour shells from the
atom positions, torch.fft, torch's own log, sin and cos).
"""
from __future__ import annotations

import copy
import dataclasses
import itertools
import math

import numpy as np
import torch

HBAR, MUB, KB = 0.658211928, 0.0000578838180661, 0.000086173324
DIP_PREF = 6.745817653234234e-07  # mu_0 mu_B^2 / nm^3 in eV
MC_TAG = 0x4D43


# ---------------------------------------------------------------------------
# the cases
def listed():
    return [
        # one evaluation of the field and the per-site energies of a small film: the
        # smallest call a driver makes, where the call itself counts
        dict(name="field_square64", kind="field", lattice="square", x=64, y=64, z=1, per=3),
        # a small film relaxed without temperature, energies recorded after every step
        dict(name="sib_square64", kind="steps", lattice="square", x=64, y=64, z=1, per=3, integrator="sib", T=0.0,
             alpha=0.3, steps=200),
        # the benchmark's lattice: three exchange shells, DMI, easy axis, field, 10 K
        dict(name="sib_triangular1024", kind="steps", lattice="triangular", x=1024, y=1024, z=1, per=3,
             integrator="sib", T=10.0, alpha=0.1, steps=20),
        # the largest, with odd sides and an open edge, the reference's own Heun scheme
        dict(name="heun_square_3001x2047", kind="steps", lattice="square", x=3001, y=2047, z=1, per=1,
             integrator="heun", T=10.0, alpha=0.1, steps=5),
        # a bulk crystal: six neighbours in three dimensions
        dict(name="sib_cubic96x96x97", kind="steps", lattice="cubic", x=96, y=96, z=97, per=7, integrator="sib",
             T=10.0, alpha=0.1, steps=10),
        # the film with dipolar interactions
        dict(name="sib_dipolar_film128x16", kind="steps", lattice="film", x=128, y=128, z=16, per=3,
             integrator="sib", T=5.0, alpha=0.1, steps=10),
        # two magnetic atoms per cell (couplings held per site)
        dict(name="sib_two_atom384", kind="steps", lattice="two_atom", x=384, y=384, z=1, per=3, integrator="sib",
             T=10.0, alpha=0.1, steps=10),
        # the host program's spins in and out, one step per call
        dict(name="host_triangular1024", kind="host", lattice="triangular", x=1024, y=1024, z=1, per=3,
             integrator="sib", T=10.0, alpha=0.1, steps=1),
        # replicas of uneven size at their own fields and temperatures, a swap round at the end
        dict(name="batch_replicas256", kind="batch", nrep=256, steps=20, alpha=0.5),
        # gradients of a trajectory for the spins, the couplings and the field map
        dict(name="adjoint_square256", kind="adjoint", x=256, y=256, steps=200, every=50, alpha=0.2),
        # Metropolis sweeps with the totals recorded after every sweep
        dict(name="mc_square1024", kind="mc", x=1024, y=1024, per=3, T=10.0, steps=10),
        # a minimum-energy path of 16 images
        dict(name="gneb_square256x16", kind="gneb", x=256, y=256, nim=16, steps=40),
    ]


def draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["field", "steps", "steps", "steps", "cubic", "film", "two_atom", "host", "batch", "adjoint",
                       "mc", "gneb"])
    alpha = round(rng.uniform(0.05, 0.5), 3)
    T = rng.choice([0.0, round(rng.uniform(1.0, 50.0), 2)])
    integrator = rng.choice(["sib", "sib", "heun", "euler"])
    if kind == "field":
        return dict(kind="field", lattice=rng.choice(["square", "triangular"]), x=size(8, 2048), y=size(8, 2048), z=1,
                    per=rng.choice([3, 3, 1, 0]))
    if kind == "steps":
        x, y = size(16, 2048), size(16, 2048)
        return dict(kind="steps", lattice=rng.choice(["square", "triangular"]), x=x, y=y, z=1,
                    per=rng.choice([3, 3, 2, 0]), integrator=integrator, T=T, alpha=alpha,
                    steps=max(5, min(200, 20_000_000 // (x * y))))
    if kind == "cubic":
        x, y, z = size(8, 96), size(8, 96), size(8, 96)
        return dict(kind="steps", lattice="cubic", x=x, y=y, z=z, per=rng.choice([7, 7, 3, 0]), integrator=integrator,
                    T=T, alpha=alpha, steps=max(5, min(50, 9_000_000 // (x * y * z))))
    if kind == "film":
        return dict(kind="steps", lattice="film", x=size(16, 128), y=size(16, 128), z=size(2, 16),
                    per=rng.choice([3, 0]), integrator=integrator, T=T, alpha=alpha, steps=10)
    if kind == "two_atom":
        return dict(kind="steps", lattice="two_atom", x=size(16, 384), y=size(16, 384), z=1, per=rng.choice([3, 0]),
                    integrator=integrator, T=T, alpha=alpha, steps=10)
    if kind == "host":
        return dict(kind="host", lattice=rng.choice(["square", "triangular"]), x=size(64, 1024), y=size(64, 1024),
                    z=1, per=3, integrator=integrator, T=T, alpha=alpha, steps=1)
    if kind == "batch":
        return dict(kind="batch", nrep=size(4, 256), steps=20, alpha=alpha)
    if kind == "adjoint":
        return dict(kind="adjoint", x=size(16, 256), y=size(16, 256), steps=size(20, 200), every=rng.choice([10, 50]),
                    alpha=alpha)
    if kind == "mc":
        per = rng.choice([3, 0])
        x, y = size(32, 1024), size(32, 1024)
        if per:  # two colours need even periodic sides
            x, y = x + x % 2, y + y % 2
        return dict(kind="mc", x=x, y=y, per=per, T=round(rng.uniform(1.0, 50.0), 2), steps=10)
    return dict(kind="gneb", x=size(16, 256), y=size(16, 256), nim=rng.randint(5, 16), steps=40)


def _deck(c):
    import matjes_b200 as mj
    from matjes_b200.deck import square_areal

    per = tuple((c.get("per", 3) >> d) & 1 for d in range(3))
    kind = c.get("lattice", "square")
    L = (c["x"], c["y"], c.get("z", 1))
    if kind == "triangular":
        d = mj.triangular(L)
        d.periodic = per
        return d
    if kind in ("film", "cubic"):
        return mj.square_film(L, Jv=1e-3, Dv=0.15e-3, Kv=-0.02e-3, Bz=0.2, a=0.25, med_z=-0.3, periodic=per,
                              dip=kind == "film")
    if kind == "two_atom":
        return mj.Deck(L=L, periodic=per, areal=square_areal(),
                       atoms=[((0, 0, 0), 1, 2.0), ((0.5, 0.5, 0), 1, 1.5), ((0.5, 0.0, -0.5), 2, 0.0)],
                       J=[(1, 1, 1, 1e-3), (1, 1, 2, 0.4e-3)], D=[(1, 1, 2, 1, 0.2e-3)],
                       K=[(1, (0, 0, 1), -0.1e-3)], B_ext=(0, 0, 0.7))
    return mj.square_film(L, Jv=1e-3, Dv=0.3e-3, Kv=-0.1e-3, Bz=0.5, periodic=per)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _spins(n, seed, ordered=False):
    """(3, n) unit spins made from the seed: uniform on the sphere, or a ferromagnet along z with thermal tilts."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    m = torch.randn((3, n), generator=g, dtype=torch.float64, device=_device())
    if ordered:
        m *= 0.2
        m[2] += 1.0
    return m / m.norm(dim=0, keepdim=True)


def _spins_of(c, seed, n):
    """A triangular lattice starts from a tilted ferromagnet with reversed disks (the benchmark's state), others random."""
    m = _spins(n, seed, ordered=c.get("lattice") == "triangular")
    if c.get("lattice") == "triangular":
        g = torch.Generator(device="cpu").manual_seed(seed)
        ctr = torch.rand((20, 2), generator=g).to(m.device) * torch.tensor([c["x"], c["y"]], device=m.device)
        y, x = torch.meshgrid(torch.arange(c["y"], device=m.device), torch.arange(c["x"], device=m.device),
                              indexing="ij")
        flip = torch.zeros((c["y"], c["x"]), dtype=torch.bool, device=m.device)
        for k in range(20):
            dx, dy = x - ctr[k, 0], y - ctr[k, 1]
            flip |= dx * dx + dy * dy - dx * dy <= 64.0
        m = torch.where(flip.reshape(1, -1), -m, m)
    return m.contiguous()


def _replicas(c, seed):
    """Sides, fields (T) and temperatures (K) of the replicas: the seed moves the fields, not the sizes."""
    rng = np.random.default_rng(2)
    L = rng.choice(np.array([32, 48, 64, 96, 128, 192, 256]), size=256)[:c["nrep"]]
    Bz = np.random.default_rng(seed).uniform(0.0, 2.0, size=c["nrep"])
    T = 50.0 ** (np.arange(c["nrep"]) / max(1, c["nrep"] - 1))
    B = np.zeros((c["nrep"], 3))
    B[:, 2] = Bz
    return np.stack([L, L], axis=1).astype(np.int32), B, T


def _path(c, seed):
    """(nim, N, 3) images from +z to -z, every interior spin turned about an axis of its own and moved a little."""
    n, nim = c["x"] * c["y"], c["nim"]
    rng = np.random.default_rng(seed)
    phi = rng.uniform(0.0, 2 * np.pi, n)
    th = np.linspace(0.0, np.pi, nim)[:, None]
    p = np.stack([np.sin(th) * np.cos(phi), np.sin(th) * np.sin(phi), np.cos(th) + 0 * phi], axis=2)
    p[1:-1] += 1e-2 * rng.uniform(-1.0, 1.0, (nim - 2, n, 3))
    return np.ascontiguousarray(p / np.linalg.norm(p, axis=2, keepdims=True))


def _gneb_deck(c):
    import matjes_b200 as mj

    return mj.square_film((c["x"], c["y"], 1), Jv=1e-3, Dv=0.4e-3, Kv=-0.2e-3, Bz=0.3, periodic=(1, 1, 0))


def _dyn(c, seed):
    return dict(integrator=c.get("integrator", "sib"), timestep=0.1, alpha=c["alpha"], temperature=c.get("T", 0.0),
                noise="philox" if c.get("T", 0.0) else "off", seed=seed)


def prepare(case, seed):
    import matjes_b200 as mj

    c, kind = case, case["kind"]
    s = dict(kind=kind, case=c)
    if kind in ("field", "steps", "host"):
        ham = mj.Hamiltonian(_deck(c))
        m = _spins_of(c, seed, ham.N)
        s.update(ham=ham, m=m)
        if kind != "field":
            s["dyn"] = mj.SpinDynamics(ham, **_dyn(c, seed))
        if kind == "host":
            s["pin"] = torch.empty((ham.N, 3), dtype=torch.float64, pin_memory=True)
            s["pin"].copy_(m.t())
            s["m"] = s["pin"].numpy()
    elif kind == "batch":
        L, B, T = _replicas(c, seed)
        b = mj.ReplicaBatch(mj.square_film((8, 8, 1), Bz=0.0), L, B, T)
        s["spins"] = _view(b)
        s["spins"].copy_(_spins(b.N, seed))
        s.update(batch=b, p=b.params(timestep=0.1, alpha=c["alpha"], noise="philox", seed=seed))
    elif kind == "adjoint":
        ham = mj.Hamiltonian(_deck(c))
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        b = torch.zeros((3, ham.N), dtype=torch.float64, device="cuda")
        b[2] = 0.5 + 0.05 * torch.randn(ham.N, generator=g, dtype=torch.float64, device="cuda")
        gT = torch.randn((3, ham.N), generator=g, dtype=torch.float64, device="cuda")
        terms = torch.tensor(mj.deck_terms(ham.deck), dtype=torch.float64)
        traj = mj.SIBTrajectory(ham, c["steps"], c["every"], timestep=0.1, alpha=c["alpha"])
        s.update(traj=traj, m=_spins(ham.N, seed).requires_grad_(), terms=terms.requires_grad_(), b=b.requires_grad_(),
                 gT=gT)
    elif kind == "mc":
        ham = mj.Hamiltonian(_deck(c))
        s.update(ham=ham, m=_spins(ham.N, seed), mc=mj.MetropolisMC(ham, seed=seed, track_totals=True))
    else:
        from matjes_b200.gneb import path_holder

        s["path"] = path_holder(_gneb_deck(c), _path(c, seed))
        s["spins"] = _view(s["path"])
    return s


def _view(batch):
    """The batch's device spins; the view keeps their owner alive."""
    t = batch.device_tensor()
    t.owner = batch
    return t


def run(state):
    s, c = state, state["case"]
    if s["kind"] == "field":
        return list(s["ham"].get_eff_field(s["m"], with_energy=True))
    if s["kind"] in ("steps", "host"):
        return [s["m"], s["dyn"].run(s["m"], c["steps"], energies=True)][::-1]
    if s["kind"] == "batch":
        E = s["batch"].step(s["p"], c["steps"], swap_every=c["steps"], energies=True)
        return [E, s["spins"]]
    if s["kind"] == "adjoint":
        mT = s["traj"](s["m"], s["terms"], s["b"])
        return [mT.detach(), *torch.autograd.grad(mT, (s["m"], s["terms"], s["b"]), s["gT"])]
    if s["kind"] == "mc":
        E, M, acc = s["mc"].sweeps(s["m"], c["steps"], c["T"], record=True)
        return [E, M, acc, s["mc"].cone, s["m"]]
    rx, ene, dene, its, fmax, _ = s["path"].gneb_path(0.3, 0.02, 1.0, 0.0, c["steps"], "I")
    return [rx, ene, dene, its, fmax, s["spins"]]


def work(case):
    """Bytes: every spin read and written once per step, sweep or iteration (field maps, gradients and outputs
    once); operations: the field's multiply-adds of each stage and about 100 for the update of a spin."""
    c = case
    nbr = {"square": 4, "triangular": 18, "cubic": 6, "film": 6, "two_atom": 8}[c.get("lattice", "square")]
    stage = 2 * 9 * min(nbr, 6) + 6 * max(0, nbr - 6) + 100
    if c["kind"] == "batch":
        n, steps = int((_replicas(c, 0)[0][:, 0].astype(np.int64) ** 2).sum()), c["steps"]
    else:
        n, steps = c["x"] * c["y"] * c.get("z", 1), c.get("steps", 1)
        n *= 2 if c.get("lattice") == "two_atom" else 1
    if c["kind"] == "field":
        return {"bytes": 56.0 * n, "flops": float(stage) * n}
    if c["kind"] == "adjoint":  # forward, then its transpose, each reading and writing one state per step
        return {"bytes": 96.0 * n * steps, "flops": 6.0 * stage * n * steps}
    if c["kind"] == "mc":
        return {"bytes": 48.0 * n * steps, "flops": float(stage) * n * steps}
    if c["kind"] == "gneb":
        return {"bytes": 48.0 * n * c["nim"] * steps, "flops": 2.0 * stage * n * c["nim"] * steps}
    if c.get("lattice") == "film":  # transforms of three components there and back on the padded grid, per stage
        pad = 1.0
        for k, d in enumerate("xyz"):
            pad *= c[d] if (c["per"] >> k) & 1 else 2 * c[d]
        fft = 2 * 3 * 2.5 * pad * math.log2(pad) + 30 * pad
        return {"bytes": 48.0 * n * steps, "flops": steps * 2.0 * (stage * n + fft)}
    two = 1.0 if c.get("integrator") == "euler" else 2.0
    return {"bytes": 48.0 * n * steps, "flops": two * stage * n * steps}


# ---------------------------------------------------------------------------
# the same results from the definitions, in 64 bits
class _Model:
    """Field and energy of a deck on spins shaped (..., 3, nmag, z, y, x)."""

    def __init__(self, deck, L=None):
        self.L = tuple(L or deck.L)  # x, y, z
        self.per = deck.periodic
        self.areal = np.asarray(deck.areal, float)
        mag = [k for k, a in enumerate(deck.atoms) if a[2] > 0]
        self.nmag = len(mag)
        pos = [np.asarray(a[0], float) @ self.areal for a in deck.atoms]
        typ = [a[1] for a in deck.atoms]
        cells = [o for o in itertools.product(range(-3, 4), repeat=3)
                 if all(self.L[d] > 1 or self.per[d] or o[d] == 0 for d in range(3))]

        def bonds(t1, t2, shell):
            out = []
            for a in range(len(pos)):
                for b in range(len(pos)):
                    if typ[a] != t1 or typ[b] != t2:
                        continue
                    for o in cells:
                        r = pos[b] + np.asarray(o, float) @ self.areal - pos[a]
                        if np.linalg.norm(r) > 1e-9:
                            out.append((np.linalg.norm(r), a, b, o))
            d = sorted({round(q[0], 6) for q in out})[shell - 1]
            return [q[1:] for q in out if abs(q[0] - d) < 1e-5]

        T = {}

        def add(a, b, o, M):
            k = (mag.index(a), mag.index(b), o)
            T[k] = T.get(k, np.zeros((3, 3))) + M

        for t1, t2, sh, v in deck.J:
            for a, b, o in bonds(t1, t2, sh):
                add(a, b, o, deck.c_H_J * v * np.eye(3))
        for t1, t2, tm, sh, v in deck.D:
            for a, b, o in bonds(t1, t2, sh):
                ra, rb = pos[a], pos[b] + np.asarray(o, float) @ self.areal
                cand = [pos[k] + np.asarray(q, float) @ self.areal for k in range(len(pos)) if typ[k] == tm
                        for q in itertools.product(range(-4, 5), range(-4, 5), (-1, 0, 1) if self.L[2] > 1 else (0,))]
                near = min(np.linalg.norm(p - (ra + rb) / 2) for p in cand)
                d = np.zeros(3)
                for p in cand:
                    if np.linalg.norm(p - (ra + rb) / 2) < near + 1e-6:
                        x = np.cross(ra - p, rb - p)
                        d += x / np.linalg.norm(x) if np.linalg.norm(x) > 1e-8 else 0.0
                if np.linalg.norm(d) > 1e-8:
                    d /= np.linalg.norm(d)
                    d[np.abs(d) < 1e-9] = 0.0
                    add(a, b, o, deck.c_H_D * v * np.array([[0, d[2], -d[1]], [-d[2], 0, d[0]], [d[1], -d[0], 0]]))
        zero = (0, 0, 0)
        for t, ax, v in deck.K:
            e = np.asarray(ax, float) / np.linalg.norm(ax)
            for k in mag:
                if typ[k] == t:
                    add(k, k, zero, deck.c_H_ani * v * np.outer(e, e))
        self.W = {}
        for (a, b, o), M in T.items():
            for k, Mk in (((a, b, o), M), ((b, a, tuple(-v for v in o)), M.T)):
                self.W[k] = self.W.get(k, 0.0) - Mk
        mu = torch.tensor([deck.atoms[k][2] for k in mag], dtype=torch.float64, device=_device())
        self.zc = -deck.c_zeeman * MUB * mu.reshape(1, -1, 1, 1, 1)
        self.b = torch.tensor(deck.B_ext, dtype=torch.float64, device=_device()).reshape(3, 1, 1, 1, 1)
        self.KF = self._dipolar(deck) if deck.dip else None

    def shape(self, m):  # (..., 3, N) -> (..., 3, nmag, z, y, x)
        x, y, z = self.L
        return m.reshape(*m.shape[:-1], z, y, x, self.nmag).movedim(-1, -4)

    def flat(self, m):
        return m.movedim(-4, -1).reshape(*m.shape[:-4], -1)

    def _shift(self, v, o):  # the value at site + o, zero past an open edge; v: (..., z, y, x)
        for d in range(3):
            if o[d] == 0:
                continue
            ax, n = v.dim() - 1 - d, self.L[d]
            if self.per[d]:
                v = torch.roll(v, -o[d], ax)
            elif abs(o[d]) >= n:
                v = torch.zeros_like(v)
            else:
                pad = list(v.shape)
                pad[ax] = abs(o[d])
                z = torch.zeros(pad, dtype=v.dtype, device=v.device)
                v = torch.cat([v.narrow(ax, o[d], n - o[d]), z], ax) if o[d] > 0 else \
                    torch.cat([z, v.narrow(ax, 0, n + o[d])], ax)
        return v

    def pair(self, m, onsite=True, unit=None):
        """The couplings' field; unit: {key: matrix} in place of the deck's own."""
        rows = [[0.0] * 3 for _ in range(self.nmag)]
        for (a, b, o), M in (self.W if unit is None else unit).items():
            if o == (0, 0, 0) and not onsite:
                continue
            s = self._shift(m.select(-4, b), o)
            for i in range(3):
                for j in range(3):
                    if torch.is_tensor(M) or M[i, j] != 0.0:
                        rows[a][i] = rows[a][i] + M[i, j] * s.select(-4, j)
        z = torch.zeros_like(m.select(-5, 0).select(-4, 0))
        return torch.stack([torch.stack([r[i] + z for r in rows], -4) for i in range(3)], -5)

    def _dipolar(self, deck):
        dev, L, per = _device(), self.L, self.per
        n = [L[d] if per[d] or L[d] == 1 else 2 * L[d] for d in range(3)]
        ar = torch.tensor(self.areal, dtype=torch.float64, device=dev)

        def axis(d):  # offset held by grid point q: 0 .. L-1, then the negative ones of an open axis
            q = torch.arange(n[d], dtype=torch.float64, device=dev)
            return torch.where(q < L[d], q, q - n[d])

        z, y, x = torch.meshgrid(axis(2), axis(1), axis(0), indexing="ij")
        valid = torch.ones_like(x)
        for d, q in ((0, x), (1, y), (2, z)):
            if n[d] != L[d]:
                valid = valid * (q > -L[d])
        K = torch.zeros((3, 3, n[2], n[1], n[0]), dtype=torch.float64, device=dev)
        span = [range(-deck.dip_cut[d], deck.dip_cut[d] + 1) if per[d] else (0,) for d in range(3)]
        for i in itertools.product(*span):
            r = [sum(ar[d, k] * (q + i[d] * L[d]) for d, q in enumerate((x, y, z))) for k in range(3)]
            r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
            inv = torch.where(r2 > 0, 1.0 / torch.sqrt(torch.where(r2 > 0, r2, torch.ones_like(r2))), 0.0)
            for a in range(3):
                for b in range(3):
                    K[a, b] += (3.0 * r[a] * r[b] * inv ** 2 - (1.0 if a == b else 0.0)) * inv ** 3
        mu = [a[2] for a in deck.atoms if a[2] > 0][0]
        self.grid = n
        return torch.fft.rfftn(-K * valid * (mu * mu * DIP_PREF * 0.5 * 0.25 / math.pi), dim=(2, 3, 4))

    def dip(self, m):  # H of m (3, 1, z, y, x)
        x, y, z = self.L
        pad = torch.zeros((3, self.grid[2], self.grid[1], self.grid[0]), dtype=torch.float64, device=m.device)
        pad[:, :z, :y, :x] = m[:, 0]
        F = torch.fft.rfftn(pad, dim=(1, 2, 3))
        H = torch.stack([sum(self.KF[a, b] * F[b] for b in range(3)) for a in range(3)])
        return torch.fft.irfftn(H, s=(self.grid[2], self.grid[1], self.grid[0]), dim=(1, 2, 3))[:, None, :z, :y, :x]

    def field(self, m, b=None):
        """(field, per-site energy, per-site share of the total energy); b: applied field (T) in m's shape."""
        zee = self.zc * (self.b if b is None else b) + torch.zeros_like(m)
        mm = self.pair(m)
        e = -0.5 * (m * mm).sum(-5) - (m * zee).sum(-5)
        if self.KF is None:
            return mm + zee, e, e
        H = self.dip(m)
        mh = (m * H).sum(-5)
        return mm + zee - 2.0 * H, e + 2.0 * mh, e + mh


def _philox(c0, c1, c2, c3, seed):
    M0, M1, W0, W1, mask = 0xD2511F53, 0xCD9E8D57, 0x9E3779B9, 0xBB67AE85, 0xFFFFFFFF
    k0, k1 = seed & mask, (seed >> 32) & mask

    def mul(M, c):
        a, b = c * (M & 0xFFFF), c * (M >> 16)
        return (b + (a >> 16)) >> 16, (a + ((b & 0xFFFF) << 16)) & mask

    for _ in range(10):
        h0, l0 = mul(M0, c0)
        h1, l1 = mul(M1, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + W0) & mask, (k1 + W1) & mask
    return c0, c1, c2, c3


def _words(n, step, stream, tag, seed):
    i = torch.arange(n, dtype=torch.int64, device=_device())
    st = stream if torch.is_tensor(stream) else torch.tensor(stream, dtype=torch.int64, device=_device())
    one = torch.zeros_like(i + st)
    return [(w.double() + 0.5) * 2.0 ** -32 for w in _philox(i + one, one + step, st + one, one + tag, seed)]


def _normals(n, step, stream, seed):
    u = _words(n, step, stream, 0, seed)
    r1, r2 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    t1, t2 = 2 * math.pi * u[1], 2 * math.pi * u[3]
    return torch.stack([r1 * torch.cos(t1), r1 * torch.sin(t1), r2 * torch.cos(t2)], -2)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-5)


def _dot(a, b):
    return (a * b).sum(-5, keepdim=True)


def _solve(m, p, H, alpha, hc):  # the Cayley solution of a SIB stage
    h = hc * (H + alpha * _cross(p / torch.sqrt(_dot(p, p)), H))
    u = _cross(m, h)
    return m + 2.0 / (1.0 + _dot(h, h)) * (u + _cross(u, h))


def _rhs(B, m, alpha):
    n = m / torch.sqrt(_dot(m, m))
    t = _cross(n, B)
    return -_cross(n, B + alpha * t) / (1.0 + alpha * alpha)


def _onto(t, m):
    return t * torch.sqrt(_dot(m, m) / _dot(t, t))


def _step(mod, m, noise, c, b=None):
    """One time step of shaped spins m; noise: the thermal field of the step or 0.0.  (new spins, energy of m)"""
    alpha, dt = c["alpha"], 0.1
    B, _, e = mod.field(m, b)
    kind = c.get("integrator", "sib")
    if kind == "sib":
        hc = -0.5 * (dt / HBAR) / (1.0 + alpha * alpha)
        mid = 0.5 * (m + _solve(m, m, B + noise, alpha, hc))
        return _solve(m, mid, mod.field(mid, b)[0] + noise, alpha, hc), e
    if kind == "euler":
        h = dt / HBAR
        D = _rhs(B, m, alpha) + (_rhs(noise, m, alpha) if torch.is_tensor(noise) else 0.0)
        return _onto(m + D * h, m), e
    h = 0.5 * dt / HBAR
    D = _rhs(B, m, alpha)
    t = _onto(m + D * h, m)
    D = 0.5 * (D + _rhs(mod.field(t, b)[0], t, alpha))
    if torch.is_tensor(noise):
        D = D + _rhs(noise, m, alpha)
    return _onto(t + D * h, t), e


def _sigma(c, T):
    dt = 0.05 if c.get("integrator") == "heun" else 0.1
    return math.sqrt(c["alpha"] * T * KB * HBAR / dt)


def _exact_steps(c, seed):
    mod = _Model(_deck(c))
    n = mod.L[0] * mod.L[1] * mod.L[2] * mod.nmag
    m = mod.shape(_spins_of(c, seed, n))
    E = []
    for k in range(c["steps"]):
        noise = mod.shape(_sigma(c, c["T"]) * _normals(n, k, 0, seed)) if c["T"] else 0.0
        m, e = _step(mod, m, noise, c)
        E.append(e.sum())
    E.append(mod.field(m)[2].sum())
    E, m = torch.stack(E[1:]), mod.flat(m)
    return [E, m] if c["kind"] == "steps" else [E.cpu().numpy(), m.t().contiguous().cpu().numpy()]


def _exact_batch(c, seed):
    import matjes_b200 as mj

    L, B, T = _replicas(c, seed)
    off = np.concatenate([[0], np.cumsum(L[:, 0].astype(np.int64) ** 2)])
    dev = _device()
    m0 = _spins(int(off[-1]), seed)
    E, out = torch.zeros(c["nrep"], dtype=torch.float64, device=dev), torch.empty_like(m0)
    cell = mj.square_film((8, 8, 1), Bz=0.0)
    for side in sorted(set(int(v) for v in L[:, 0])):  # the replicas of one size together
        r = [k for k in range(c["nrep"]) if L[k, 0] == side]
        mod = _Model(cell, (side, side, 1))
        mod.per = (1, 1, 0)
        m = mod.shape(torch.stack([m0[:, off[k]:off[k + 1]] for k in r]))
        b = torch.tensor(B[r], device=dev).reshape(len(r), 3, 1, 1, 1, 1)
        sg = torch.tensor([_sigma(c, T[k]) for k in r], dtype=torch.float64, device=dev).reshape(-1, 1, 1)
        stream = torch.tensor(r, dtype=torch.int64, device=dev).reshape(-1, 1)
        for k in range(c["steps"]):
            m, _ = _step(mod, m, mod.shape(sg * _normals(side * side, k, stream, seed)), c, b)
        e = mod.field(m, b)[2].reshape(len(r), -1).sum(1)
        f = mod.flat(m)
        for q, k in enumerate(r):
            E[k], out[:, off[k]:off[k + 1]] = e[q], f[q]
    return [E, out]


def _exact_adjoint(c, seed):
    """torch autograd through the same steps, the couplings as sums of the terms' unit matrices."""
    from torch.utils.checkpoint import checkpoint

    deck = _deck(c)
    mod, n, dev = _Model(deck), deck.nsites, _device()
    g = torch.Generator(device=dev).manual_seed(seed + 1)
    b = torch.zeros((3, n), dtype=torch.float64, device=dev)
    b[2] = 0.5 + 0.05 * torch.randn(n, generator=g, dtype=torch.float64, device=dev)
    gT = torch.randn((3, n), generator=g, dtype=torch.float64, device=dev)
    none = dict(J=[], D=[], K=[])
    units = [_Model(dataclasses.replace(deck, **{**none, k: [t[:-1] + (1.0,)]})).W for k in ("J", "D", "K")
             for t in getattr(deck, k)]
    terms = torch.tensor([t[-1] for k in ("J", "D", "K") for t in getattr(deck, k)], dtype=torch.float64, device=dev)
    m0 = _spins(n, seed).requires_grad_()
    terms, b = terms.requires_grad_(), b.requires_grad_()

    def part(m, b, terms, k):
        W = {}
        for t, u in zip(terms, units):
            for key, M in u.items():
                W[key] = W.get(key, 0.0) + t * torch.tensor(M, dtype=torch.float64, device=dev)
        own = copy.copy(mod)
        own.pair = lambda v: mod.pair(v, unit=W)
        for _ in range(k):
            m, _e = _step(own, m, 0.0, c, b)
        return m

    m, bs, left = mod.shape(m0), mod.shape(b), c["steps"]
    while left > 0:
        m = checkpoint(part, m, bs, terms, min(20, left), use_reentrant=False)
        left -= 20
    mT = mod.flat(m)
    grads = torch.autograd.grad(mT, (m0, terms, b), gT)
    return [mT.detach(), grads[0], grads[1].cpu(), grads[2]]


def _exact_mc(c, seed):
    """Colour by colour (x + y) mod 2, proposals uniform in the cone about the spin, the cone updated per sweep."""
    mod = _Model(_deck(c))
    n, kT = c["x"] * c["y"], c["T"] * KB
    m = mod.shape(_spins(n, seed))
    W0 = torch.tensor(mod.W[(0, 0, (0, 0, 0))], dtype=torch.float64, device=m.device)
    y, x = torch.meshgrid(torch.arange(c["y"], device=m.device), torch.arange(c["x"], device=m.device), indexing="ij")
    colour, cone, total, tried = (x + y) % 2, math.pi, 0, 0
    zee = mod.zc * mod.b + torch.zeros_like(m)
    on = lambda v: torch.einsum("ij,jazyx->iazyx", W0, v)  # noqa: E731
    Es, Ms = [], []
    for k in range(c["steps"]):
        u = [w.reshape(1, 1, 1, c["y"], c["x"]) for w in _words(n, k, 0, MC_TAG, seed)]
        for col in (0, 1):
            P = mod.pair(m, onsite=False)
            ct = u[0] + math.cos(cone) * (1.0 - u[0])
            st = torch.sqrt(1.0 - ct * ct)
            sx, sy, sz = m[0:1], m[1:2], m[2:3]
            rxy2 = sx * sx + sy * sy
            sti, far = torch.sqrt(rxy2), ~(rxy2 < 0.00001)
            safe = torch.where(far, sti, torch.ones_like(sti))
            cpi, spi = torch.where(far, sx / safe, 1.0), torch.where(far, sy / safe, 0.0)
            sph, cph = torch.sin(2 * math.pi * u[1]), torch.cos(2 * math.pi * u[1])
            t = st * sph * sz + ct * sti
            new = torch.cat([-st * cph * spi + t * cpi, st * cph * cpi + t * spi, -st * sph * sti + ct * sz])
            new = new / torch.sqrt(_dot(new, new))
            d = new - m
            dE = -_dot(d, P) - 0.5 * (_dot(new, on(new)) - _dot(m, on(m))) - _dot(d, zee)
            acc = ((dE < 0) | (u[2] < torch.exp(torch.clamp(-dE / kT, min=-200.0)))) & (colour == col)
            m = torch.where(acc, new, m)
            total += int(acc.sum())
        Es.append(mod.field(m)[2].sum())
        Ms.append(m.reshape(3, -1).sum(1))
        tried += n
        rate, inc = total / tried, 1e-4 * n
        if rate > 0.5 and cone < math.pi:
            cone = min(math.pi, cone + inc)
        elif rate < 0.5 and cone > 0.01:
            cone = max(0.01, cone - inc)
    return [torch.stack(Es), torch.stack(Ms), total, cone, mod.flat(m)]


def _exact_gneb(c, seed):
    """Velocity projection on the path's forces, the tangents weighted by the images' energies."""
    mod, nim, dt, spring = _Model(_gneb_deck(c)), c["nim"], 0.02, 0.3
    p = torch.tensor(_path(c, seed), device=_device()).transpose(1, 2).contiguous()
    m = mod.shape(p)

    def tang(v, q):
        v = v - _dot(v, q) * q
        return v / torch.sqrt((v * v).sum())

    def force(m):
        B, _, e = mod.field(m)
        F = B - _dot(B, m) * m
        E = e.reshape(nim, -1).sum(1)
        cr = _cross(m[:-1], m[1:])
        ang = torch.atan2(torch.sqrt(_dot(cr, cr)), _dot(m[:-1], m[1:]))
        pl = torch.cat([E.new_zeros(1), torch.cumsum(torch.sqrt((ang ** 2).reshape(nim - 1, -1).sum(1)), 0)])
        G, along = F.clone(), [None] * nim
        for i in range(nim):
            simple = tang(m[min(i + 1, nim - 1)] - m[max(i - 1, 0)], m[i])
            along[i] = (F[i] * simple).sum()
            if i in (0, nim - 1):
                continue
            u1, u2, u3 = (float(E[i + q]) for q in (-1, 0, 1))
            hi, lo = max(abs(u3 - u2), abs(u1 - u2)), min(abs(u3 - u2), abs(u1 - u2))
            wp, wm = (1.0, 0.0) if u3 > u2 > u1 else (0.0, 1.0) if u1 > u2 > u3 else (hi, lo) if u3 > u1 else (lo, hi)
            t = tang(wp * (m[i + 1] - m[i]) + wm * (m[i] - m[i - 1]), m[i])
            G[i] = F[i] - t * (F[i] * t).sum() + spring * (pl[i + 1] + pl[i - 1] - 2.0 * pl[i]) * t
        return F, G, E, pl, torch.stack(along)

    def turn(v, ax, cs, sn):
        return v * cs + sn * _cross(v, ax) + (1.0 - cs) * _dot(ax, v) * ax

    F, G, E, pl, along = force(m)
    e0 = E[0].clone()
    inner = slice(1, nim - 1)
    v, F1 = torch.zeros_like(m), G
    for _ in range(c["steps"]):
        f = F1[inner]
        ax = _cross(m[inner], f)
        na = torch.sqrt(_dot(ax, ax))
        ax = ax / torch.where(na > 0, na, torch.ones_like(na))
        r = m[inner] + v[inner] * dt + 0.5 * f * dt * dt
        r = r / torch.sqrt(_dot(r, r))
        cr = _cross(m[inner], r)
        ang = torch.atan2(torch.sqrt(_dot(cr, cr)), _dot(m[inner], r))
        cs, sn = torch.cos(ang), torch.sin(ang)
        vel, old = turn(v[inner], ax, cs, sn), turn(f, ax, cs, sn)
        m = torch.cat([m[:1], r, m[-1:]])
        F, G, E, pl, along = force(m)
        F2 = torch.cat([torch.zeros_like(m[:1]), G[inner], torch.zeros_like(m[:1])])  # the ends are held
        vel = torch.cat([v[:1], vel + 0.5 * (old + F2[inner]) * dt, v[-1:]])
        fv, ff = (vel * F2).sum(), (F2 * F2).sum()
        v = F2 * torch.clamp(fv / ff, min=0.0)
        F1 = F2
    dene = -torch.cat([E.new_zeros(1), along[inner], E.new_zeros(1)])
    images = mod.flat(m).movedim(1, 0).reshape(3, -1).contiguous()
    return [pl.cpu().numpy(), (E - e0).cpu().numpy(), dene.cpu().numpy(), c["steps"], float(F1.abs().max()), images]


def exact(case, seed):
    c = case
    if c["kind"] == "field":
        mod = _Model(_deck(c))
        B, e, _ = mod.field(mod.shape(_spins_of(c, seed, c["x"] * c["y"] * c["z"])))
        return [mod.flat(B), mod.flat(e[None])[0]]
    if c["kind"] in ("steps", "host"):
        return _exact_steps(c, seed)
    if c["kind"] == "batch":
        return _exact_batch(c, seed)
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, seed)
    if c["kind"] == "mc":
        return _exact_mc(c, seed)
    return _exact_gneb(c, seed)
