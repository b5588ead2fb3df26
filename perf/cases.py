"""Timed cases of the halo-finding path, each a call that a program using the package makes.

listed() names twelve cases over six kinds of call; draw() gives others of the same ranges:

  fof         FoF labels and the groups of a star snapshot held on the GPU
  unbind      batched iterative unbinding of a catalogue of haloes held on the GPU
  find        the one-call pipeline (FoF, groups, unbinding) on a snapshot held on the GPU
  potential   the drop-in of the Fortran potential on host arrays (ram-pressure stripping,
              most-bound search, escape cut)
  gradient    softened potential energy of a gas halo and its gradients through autograd
  properties  the per-halo property loop of the main script on host arrays

The inputs are Plummer spheres with power-law sizes, unbound contaminants and a uniform
background, or an NFW gas halo with stars, in the units of the package (Mpc, km/s, Msun).
"""
import math

import numpy as np
import torch

from pyhalma_gb300 import fof, halo_gas, halo_properties
from pyhalma_gb300.autograd import softened_potential
from pyhalma_gb300.unbinding import UnbindOptions, find_haloes, unbind_batched

G_MPC = 4.3e-9            # (km/s)^2 Mpc / Msun
EPS = 1e-4                # softening, Mpc
LL = 1.5e-3               # linking length, Mpc
PARTICLE_MASS = 4e6       # Msun
CONTAMINANTS = 0.15       # share of a halo's members that are not bound to it
MAX_ITER = 30
EXACT_PAIRS = 6e9         # exact() sums at most so many pairs in 64 bits


def listed():
    return [
        # a small zoom or test box: the call is launches and round trips
        {"name": "fof_5k", "kind": "fof", "n": 5_000, "haloes": 8, "alpha": 0.0, "box": 2.0, "ll": LL, "minp": 2},
        # the repository's 2e6-particle, 500-sphere snapshot
        {"name": "fof_2m", "kind": "fof", "n": 2_000_000, "haloes": 500, "alpha": 0.0, "box": 10.0, "ll": LL,
         "minp": 50},
        # a large snapshot with the power-law haloes of the 5e7-particle one, 0.4 of its size
        {"name": "fof_20m", "kind": "fof", "n": 20_000_000, "haloes": 8_000, "alpha": 0.575, "box": 74.0, "ll": LL,
         "minp": 50},
        # the haloes of a small box
        {"name": "unbind_24", "kind": "unbind", "haloes": 24, "lo": 50, "hi": 1_000, "alpha": 0.0},
        # the haloes of the 2e6-particle snapshot
        {"name": "unbind_500", "kind": "unbind", "haloes": 500, "lo": 50, "hi": 30_000, "alpha": 0.0},
        # half of the batched catalogue (dN/dlogN ~ 1/N on [50, 2e5])
        {"name": "unbind_10k", "kind": "unbind", "haloes": 10_000, "lo": 50, "hi": 200_000, "alpha": 1.0},
        # one snapshot from positions to bound haloes
        {"name": "find_1m", "kind": "find", "n": 1_000_000, "haloes": 300, "alpha": 0.0, "box": 8.0, "ll": LL,
         "minp": 50},
        # gas cells of an ordinary galaxy against a sampled source family, as the RPS block calls it
        {"name": "potential_2k_x_20k", "kind": "potential", "targets": 2_000, "sources": 20_000,
         "mode": "reference"},
        # a massive halo: tens of thousands of cells against all its particles
        {"name": "potential_40k_x_100k", "kind": "potential", "targets": 40_000, "sources": 100_000,
         "mode": "reference"},
        # accelerations and dE/dm of a dwarf and of a massive gas halo
        {"name": "gradient_4k", "kind": "gradient", "gas": 3_000, "stars": 1_001},
        {"name": "gradient_200k", "kind": "gradient", "gas": 160_000, "stars": 40_000},
        # the property loop over the haloes of an ordinary snapshot
        {"name": "properties_120", "kind": "properties", "haloes": 120, "lo": 50, "hi": 20_000, "alpha": 0.0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fof", "unbind", "find", "potential", "gradient", "properties"])
    if kind in ("fof", "find"):
        n = _log_uniform(rng, 4_000, 20_000_000 if kind == "fof" else 1_500_000)
        haloes = max(4, int(n / math.exp(rng.uniform(math.log(1_500), math.log(6_000)))))
        box = 10.0 * (n / 2e6) ** (1.0 / 3.0) * math.exp(rng.uniform(0.0, math.log(3.0)))
        return {"kind": kind, "n": n, "haloes": haloes, "alpha": rng.choice([0.0, 0.575]), "box": round(box, 3),
                "ll": round(LL * rng.uniform(0.7, 1.3), 7), "minp": rng.choice([2, 20, 50])}
    if kind == "unbind":
        while True:
            case = {"kind": kind, "haloes": _log_uniform(rng, 1, 10_000), "lo": rng.choice([32, 50, 333]),
                    "hi": _log_uniform(rng, 600, 200_000), "alpha": rng.choice([0.0, 0.575, 1.0])}
            c = _counts(case).astype(np.float64)
            if c.sum() < 8e6 and (c * c).sum() < 1.2e11:
                return case
    if kind == "potential":
        return {"kind": kind, "targets": _log_uniform(rng, 60, 60_000), "sources": _log_uniform(rng, 1_000, 100_000),
                "mode": rng.choice(["reference", "reference", "reference", "fast"])}
    if kind == "gradient":
        gas = _log_uniform(rng, 500, 160_000)
        return {"kind": kind, "gas": gas, "stars": max(1, int(gas * rng.uniform(0.02, 0.4)))}
    while True:
        case = {"kind": kind, "haloes": _log_uniform(rng, 1, 600), "lo": 50, "hi": _log_uniform(rng, 600, 40_000),
                "alpha": rng.choice([0.0, 0.575])}
        if _counts(case).sum() < 1_200_000:
            return case


# ---- inputs --------------------------------------------------------------------------------
def _counts(case):
    """Halo sizes: quantiles of dN/dlogN ~ N^-alpha on [lo, hi]."""
    lo, hi, a, k = case.get("lo", 50), case.get("hi", 200_000), case["alpha"], case["haloes"]
    q = (np.arange(k) + 0.5) / k
    if a == 0.0:
        c = lo * (hi / lo) ** q
    else:
        c = (lo ** -a - q * (lo ** -a - hi ** -a)) ** (-1.0 / a)
    return np.maximum(1, np.round(c)).astype(np.int64)


class _Random:
    """Random numbers on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def unit(self, n):
        v = self.normal(n, 3)
        return v / v.norm(dim=1, keepdim=True).clamp_min(1e-300)


def _spheres(r, counts, centres):
    """Plummer spheres with contaminants; positions [n, 3] in Mpc, velocities [n, 3] in km/s."""
    counts = torch.as_tensor(counts, device="cuda")
    k, n = counts.shape[0], int(counts.sum())
    of = torch.repeat_interleave(torch.arange(k, device="cuda"), counts, output_size=n)
    mass = counts.double() * PARTICLE_MASS
    a = (2e-3 * (mass / 1e10) ** (1.0 / 3.0))[of]
    m = mass[of]
    stray = r.uniform(n) < CONTAMINANTS
    u = 1e-6 + r.uniform(n) * (0.999 - 1e-6)
    rad = torch.where(stray, 3.0 * a * u ** (1.0 / 3.0), a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0))
    pos = centres[of] + rad[:, None] * r.unit(n)
    sigma = torch.sqrt(G_MPC * m / (6.0 * a))
    escape = torch.sqrt(2.0 * G_MPC * m / torch.sqrt(rad * rad + a * a))
    vel = torch.where(stray[:, None], (3.0 * escape)[:, None] * r.unit(n), sigma[:, None] * r.normal(n, 3))
    return pos, vel + (200.0 * r.normal(k, 3))[of]


def _sizes(case, r):
    """The sizes in an order of the seed's own."""
    return _counts(case)[r.uniform(case["haloes"]).argsort().cpu().numpy()]


def _columns(t):
    return [t[:, d].contiguous() for d in range(3)]


def _catalogue(case, seed):
    r = _Random(seed)
    counts = _sizes(case, r)
    centres = 100.0 * (r.uniform(case["haloes"], 3) - 0.5)
    pos, vel = _spheres(r, counts, centres)
    off = torch.zeros(len(counts) + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.as_tensor(counts, device="cuda").cumsum(0)
    mass = torch.full((pos.shape[0],), PARTICLE_MASS, dtype=torch.float64, device="cuda")
    return off, [*_columns(pos), *_columns(vel), mass]


def _snapshot(case, seed):
    r = _Random(seed)
    n, box = case["n"], case["box"]
    c = _sizes(case, r).astype(np.float64)
    counts = np.maximum(1, np.floor(c * (0.88 * n / c.sum()))).astype(np.int64)
    centres = (box - 0.4) * (r.uniform(case["haloes"], 3) - 0.5)
    pos, vel = _spheres(r, counts, centres)
    rest = n - pos.shape[0]
    pos = torch.cat([pos, box * (r.uniform(rest, 3) - 0.5)])
    vel = torch.cat([vel, 300.0 * r.normal(rest, 3)])
    order = torch.randperm(n, generator=r.g, device="cuda") if n < 100_000 else None   # small files come unsorted
    if order is not None:
        pos, vel = pos[order], vel[order]
    return [*_columns(pos), *_columns(vel), torch.full((n,), PARTICLE_MASS, dtype=torch.float64, device="cuda")]


def _gas_halo(r, n_gas, n_stars):
    """NFW gas cells (concentration 8, 150 kpc, lognormal masses) and a Plummer body of stars."""
    x = torch.logspace(-5, math.log10(8.0), 4096, device="cuda", dtype=torch.float64)
    mu = torch.log1p(x) - x / (1.0 + x)
    u = r.uniform(n_gas) * mu[-1]
    i = torch.searchsorted(mu, u).clamp(1, 4095)
    rad = x[i - 1] + (x[i] - x[i - 1]) * ((u - mu[i - 1]) / (mu[i] - mu[i - 1]))
    gas = (0.15 / 8.0) * rad[:, None] * r.unit(n_gas)
    a = 2e-3 * (n_stars * 1e5 / 1e10) ** (1.0 / 3.0)
    v = 1e-6 + r.uniform(n_stars) * (0.999 - 1e-6)
    stars = (a / torch.sqrt(v ** (-2.0 / 3.0) - 1.0))[:, None] * r.unit(n_stars)
    mass = torch.cat([torch.exp(math.log(1e5) + r.normal(n_gas)),
                      torch.full((n_stars,), 1e5, dtype=torch.float64, device="cuda")])
    return torch.cat([gas, stars]), mass


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fof":
        return {"case": case, "x": _snapshot(case, seed)[:3]}
    if kind == "find":
        return {"case": case, "x": _snapshot(case, seed)}
    if kind == "unbind":
        off, cols = _catalogue(case, seed)
        return {"case": case, "off": off, "x": cols}
    if kind == "potential":
        # all sources of the halo; the targets are its gas cells, which are sources too
        r = _Random(seed)
        gas = min(case["targets"], case["sources"] // 2)
        pos, mass = _gas_halo(r, case["targets"], case["sources"] - gas)
        src = torch.cat([pos[:gas], pos[case["targets"]:]]) + 3.0
        tgt = pos[:case["targets"]] + 3.0
        m = torch.cat([mass[:gas], mass[case["targets"]:]])
        cols = [m, *_columns(src), *_columns(tgt)]
        return {"case": case, "x": [c.cpu().numpy() for c in cols]}
    if kind == "gradient":
        r = _Random(seed)
        pos, mass = _gas_halo(r, case["gas"], case["stars"])
        return {"case": case, "x": [c.float().requires_grad_(True) for c in (*_columns(pos), mass)]}
    off, cols = _catalogue(case, seed)
    off = off.cpu().numpy()
    order = torch.randperm(int(off[-1]), generator=_Random(seed + 1).g, device="cuda")   # particles in file order
    place = torch.empty_like(order)
    place[order] = torch.arange(order.shape[0], device="cuda")
    cols = [c[order].cpu().numpy() for c in cols]
    place = place.cpu().numpy()
    groups = [np.sort(place[off[h]:off[h + 1]]) for h in range(len(off) - 1)]
    about = []
    for g in groups:
        c = [float(cols[d][g].mean()) for d in range(3)]
        far = math.sqrt(max(sum((cols[d][g] - c[d]) ** 2 for d in range(3))))
        about.append([*c, PARTICLE_MASS * len(g), far])
    return {"case": case, "x": cols, "groups": groups, "about": [np.array(a) for a in zip(*about)]}


# ---- one pass ------------------------------------------------------------------------------
def _rows(t, k):
    """t with zeros after it up to k rows: the number of groups depends on the seed, an output's shape does not."""
    return torch.cat([t, t.new_zeros(k - t.shape[0], *t.shape[1:])])


def run(state):
    case, x = state["case"], state["x"]
    kind = case["kind"]
    if kind == "fof":
        labels = fof.fof_labels(*x, case["ll"])
        offsets, members = fof.fof_groups(labels, case["minp"])
        return {"labels": labels, "offsets": _rows(offsets, case["n"] // 2 + 2), "members": _rows(members, case["n"])}
    if kind == "unbind":
        bound, haloes, _ = unbind_batched(state["off"], *x, UnbindOptions(eps=EPS, max_iter=MAX_ITER))
        return {"bound": bound, "haloes": haloes}
    if kind == "find":
        c = find_haloes(*x, case["ll"], case["minp"], UnbindOptions(eps=EPS, max_iter=MAX_ITER))
        k = case["n"] // case["minp"] + 2
        return {"labels": c.labels, "bound": c.bound, "offsets": _rows(c.offsets, k),
                "members": _rows(c.members, case["n"]), "haloes": _rows(c.haloes, k)}
    if kind == "potential":
        return halo_gas.bf_potential(*x, mode=case["mode"])
    if kind == "gradient":
        sx, sy, sz, m = x
        k = case["gas"]
        phi = softened_potential(sx, sy, sz, m, sx[:k], sy[:k], sz[:k], EPS)
        energy = -(m[:k] * phi).sum()
        return [phi.detach(), *torch.autograd.grad(energy, x)]
    return halo_properties.property_loop(state["groups"], *x, *state["about"], LL)


# ---- what a pass cannot do without -----------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "fof":   # positions in; labels, members and offsets out
        return {"bytes": 36.0 * case["n"], "flops": 8.0 * case["n"]}
    if kind in ("unbind", "find"):
        c = _counts(case).astype(np.float64)
        if kind == "find":
            c = c * (0.88 * case["n"] / c.sum())
        n = case.get("n", c.sum())
        # 14 operations a pair, each pair once for both particles, and the removed ones again
        flops = 14.0 * (0.5 + CONTAMINANTS) * (c * c).sum()
        return {"bytes": (57.0 if kind == "unbind" else 65.0) * n + 96.0 * len(c), "flops": flops}
    if kind == "potential":
        return {"bytes": 16.0 * case["sources"] + 16.0 * case["targets"],
                "flops": 13.0 * case["sources"] * case["targets"]}
    if kind == "gradient":   # forward 12 operations a pair, backward 24 for both of its ends
        n = case["gas"] + case["stars"]
        return {"bytes": 36.0 * n, "flops": 36.0 * n * case["gas"]}
    n = float(_counts(case).sum())
    return {"bytes": 60.0 * n, "flops": 150.0 * n}


# ---- the same in 64 bits ---------------------------------------------------------------------
def _blocks(nt, ns):
    step = max(1, int(4e7 // max(ns, 1)))
    return [slice(b, min(nt, b + step)) for b in range(0, nt, step)]


def _exact_unbind(pos, vel, m, out):
    """One halo: escape cut repeated until a pass removes nothing."""
    bound = torch.ones(m.shape[0], dtype=torch.bool, device="cuda")
    for it in range(1, MAX_ITER + 1):
        p, v, w = pos[bound], vel[bound], m[bound]
        bulk = (w[:, None] * v).sum(0) / w.sum()
        phi = torch.empty_like(w)
        for s in _blocks(len(w), len(w)):
            r2 = ((p[s, None, 0] - p[None, :, 0]) ** 2 + (p[s, None, 1] - p[None, :, 1]) ** 2
                  + (p[s, None, 2] - p[None, :, 2]) ** 2 + EPS * EPS)
            phi[s] = torch.rsqrt(r2) @ w
        phi -= w / EPS
        kin = 0.5 * ((v - bulk) ** 2).sum(1)
        keep = ~(kin - G_MPC * phi > 0.0)
        e_kin, e_pot = (w * kin)[keep].sum(), -0.5 * G_MPC * (w * phi)[keep].sum()
        bound[bound.clone()] = keep
        if bool(keep.all()) or not bool(keep.any()):
            break
    w = m[bound]
    total = w.sum()
    centre, bulk = ((w[:, None] * t[bound]).sum(0) / total if total > 0 else torch.zeros(3, device="cuda",
                    dtype=torch.float64) for t in (pos, vel))
    out[:] = torch.stack([total, *centre, *bulk, torch.tensor(float(len(w)), device="cuda", dtype=torch.float64),
                          torch.tensor(float(it), device="cuda", dtype=torch.float64), e_kin, e_pot])


def _exact_properties(state):
    x, y, z, vx, vy, vz, m = state["x"]
    names = halo_properties_names()
    table = {k: np.zeros(len(state["groups"])) for k in names}
    for h, g in enumerate(state["groups"]):
        cx, cy, cz, mass, _ = (a[h] for a in state["about"])
        r = np.stack([x[g] - cx, y[g] - cy, z[g] - cz], 1)
        v = np.stack([vx[g], vy[g], vz[g]], 1)
        w = m[g]
        bulk = (w[:, None] * v).sum(0) / mass
        v = v - bulk
        for name, axes in (("rad05", (0, 1, 2)), ("rad05_x", (1, 2)), ("rad05_y", (0, 2)), ("rad05_z", (0, 1))):
            d = np.sqrt((r[:, axes] ** 2).sum(1))
            order = np.argsort(d, kind="stable")
            first = int(np.argmax(np.cumsum(w[order]) > 0.5 * mass))
            table[name][h] = d[order][max(first - 1, 0)]
        j = np.array([(w * (r[:, 1] * v[:, 2] - r[:, 2] * v[:, 1])).sum(),
                      (w * (r[:, 2] * v[:, 0] - r[:, 0] * v[:, 2])).sum(),
                      (w * (r[:, 0] * v[:, 1] - r[:, 1] * v[:, 2])).sum()]) / mass
        for d, name in enumerate("xyz"):
            table["velocities_" + name][h] = bulk[d]
            table["specific_angular_momentum_" + name][h] = j[d]
        table["specific_angular_momentum"][h] = np.sqrt((j * j).sum())
        inside = np.sqrt((r ** 2).sum(1)) < table["rad05"][h]
        table["sig_3D"][h] = math.sqrt((v[inside] ** 2).sum() / 3.0 / max(1, inside.sum()))
        tensor = (w[:, None, None] * r[:, :, None] * r[:, None, :]).sum(0) / w.sum()
        axes = np.sqrt(np.sort(np.linalg.eigvalsh(tensor))[::-1])
        for d, name in enumerate(("s_axis_major", "s_axis_intermediate", "s_axis_minor")):
            table[name][h] = axes[d]
    return {k: table[k] if k in EXACT_PROPERTIES else None for k in names}


EXACT_PROPERTIES = {"rad05", "rad05_x", "rad05_y", "rad05_z", "velocities_x", "velocities_y", "velocities_z",
                    "specific_angular_momentum_x", "specific_angular_momentum_y", "specific_angular_momentum_z",
                    "specific_angular_momentum", "sig_3D", "s_axis_major", "s_axis_intermediate", "s_axis_minor"}


def halo_properties_names():
    return list(EXACT_PROPERTIES) + ["tully_fisher_velocities", "kinematic_morphologies", "sig_1D_x", "sig_1D_y",
                                     "sig_1D_z", "vsigma", "lambda_ensellem"]


def exact(case, seed):
    """The floating outputs of run() in 64 bits (None for whole numbers, and where the pairs are too many)."""
    kind = case["kind"]
    if kind in ("fof", "find"):
        return None
    if kind == "unbind":
        c = _counts(case).astype(np.float64)
        if (c * c).sum() > EXACT_PAIRS / 4 or len(c) > 600:
            return None
        off, cols = _catalogue(case, seed)
        pos, vel, m = torch.stack(cols[:3], 1), torch.stack(cols[3:6], 1), cols[6]
        table = torch.zeros(case["haloes"], 11, dtype=torch.float64, device="cuda")
        o = off.tolist()
        for h in range(case["haloes"]):
            s = slice(o[h], o[h + 1])
            _exact_unbind(pos[s], vel[s], m[s], table[h])
        return {"bound": None, "haloes": table}
    if kind == "potential":
        if case["targets"] * case["sources"] > EXACT_PAIRS:
            return None
        # the entry point takes single-precision inputs: the sum is exact for those
        m, x, y, z, tx, ty, tz = (torch.as_tensor(c, device="cuda").float().double() for c in prepare(case, seed)["x"])
        phi = torch.empty_like(tx)
        for s in _blocks(len(tx), len(x)):
            dx, dy, dz = x - tx[s, None], y - ty[s, None], z - tz[s, None]
            term = torch.where((dx != 0) & (dy != 0) & (dz != 0), 1.0 / torch.sqrt(dx * dx + dy * dy + dz * dz), 0.0)
            phi[s] = term @ m
        return phi.cpu().numpy()
    if kind == "gradient":
        n, k = case["gas"] + case["stars"], case["gas"]
        if n * k > 6 * EXACT_PAIRS:
            return None
        x, y, z, m = (c.detach().double() for c in prepare(case, seed)["x"])
        phi = torch.zeros(k, dtype=torch.float64, device="cuda")
        gm = torch.zeros(n, dtype=torch.float64, device="cuda")
        force = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
        for s in _blocks(k, n):
            d = [c - c[s, None] for c in (x, y, z)]
            ri = torch.rsqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + EPS * EPS)
            phi[s] = ri @ m
            gm -= m[s] @ ri
            ri = ri ** 3
            for q in range(3):
                t = ri * d[q]
                force[q] += m * (m[s] @ t)
                force[q][s] -= m[s] * (t @ m)
        gm[:k] -= phi
        return [phi, *force, gm]
    return _exact_properties(prepare(case, seed))
