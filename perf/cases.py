"""The workloads this framework is timed on.

Every case is a call a user's program makes through the package's public
entry points: resident MD steps (MdState), the host-buffer step, trajectory
output, batched and served members (MdBatch, Server), one force evaluation,
and the flat-pair drop-in (gpu_interface).  Sizes run from 512 waters to
some 320,000 sites, with ragged water counts, boxes that are not cubes, and
the options that runs use in earnest (thermostats, barostat, constraints,
Ewald corrections, alchemical decoupling).

Systems are made from the seed alone: a unit cell (waters, optionally one
ff19SB peptide and salt) is relaxed here in float64, tiled to the case's
size, displaced by thermal amounts and given Maxwell-Boltzmann velocities.
The float64 answers of ``exact`` are plain torch: every site pair in the
cutoff, smooth PME, bonded terms, one rigid-body Verlet step.
"""
import functools
import math

import numpy as np
import torch

from dynamics_b200 import gpu_interface, md, peptide, serve, synth

DT = 0.002               # ps
SKIN = 4.0               # list skin of the flat-pair layer (the reference's default)
TEMP = 300.0
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(name, kind, waters, rho, residues=0, tiles=(1, 1, 1), drop=0, rc=10.0, integ="csvr", steps=20,
          salt=0.0, barostat=False, corrected=False, rattle=False, spme_every=2, lam=-1.0):
    """waters, rho, residues, salt: waters, their density per cubic angstrom,
    peptide length and NaCl molarity of the unit cell; tiles: its copies per
    axis; drop: waters taken out after tiling; lam: alchemical lambda of the
    first peptide (< 0: none)."""
    return {"name": name, "kind": kind, "waters": waters, "rho": rho, "residues": residues, "tx": tiles[0],
            "ty": tiles[1], "tz": tiles[2], "drop": drop, "rc": rc, "integ": integ, "steps": steps, "salt": salt,
            "barostat": barostat, "corrected": corrected, "rattle": rattle, "spme_every": spme_every, "lam": lam}


def listed():
    return [
        # the smallest simulation: a small water box under Langevin dynamics,
        # read out every 20 steps; launches and latency count
        _case("water_512", "step", 512, 0.0336, integ="langevin"),
        # a free-energy window: one of two peptides half decoupled, an odd water count
        _case("ti_window_1733", "step", 880, 0.0334, residues=10, tiles=(2, 1, 1), drop=27, rc=9.0,
              integ="langevin", lam=0.25),
        # an ordinary production run: ~32k sites, trajectory frames every 10 steps
        _case("traj_32k", "traj", 975, 0.0327, residues=5, tiles=(2, 2, 2), rc=9.0),
        # constant-energy quality: corrections, RATTLE, SPME on every step
        _case("nve_12k", "step", 1000, 0.0334, residues=10, tiles=(3, 1, 1), drop=101, rc=9.0, integ="nve",
              corrected=True, rattle=True, spme_every=1),
        # the large solvated system: peptides, 0.15 M NaCl, ~100k sites, pressure coupling
        _case("npt_100k", "step", 889, 0.0255, residues=11, tiles=(3, 3, 3), salt=0.15, barostat=True),
        # the largest: ~320k sites of water
        _case("water_80k", "step", 1000, 0.0255, tiles=(5, 4, 4), drop=333, steps=10),
        # a program that keeps its state on the host and steps on the GPU
        _case("host_step_24k", "host", 889, 0.0255, tiles=(3, 3, 3), integ="nve", steps=1),
        # one force evaluation read back (analysis, another integrator)
        _case("forces_32k", "forces", 975, 0.0327, residues=5, tiles=(2, 2, 2), rc=9.0, corrected=True),
        # the flat-pair drop-in between list rebuilds: 14 M pairs
        _case("pairs_8k", "pairs", 975, 0.0327, residues=5, tiles=(2, 2, 2), rc=9.0),
        # ... and a step that rebuilds its list, at the smallest size
        _case("rebuild_512", "rebuild", 480, 0.0336, residues=6),
        # 64 systems of 512 to 8000 waters advanced together
        dict(_case("batch_64", "batch", 0, 0.0334, rc=9.0, integ="langevin", steps=10), members=64),
        # requests that join and leave between rounds
        dict(_case("serve_6", "serve", 0, 0.0334, rc=9.0, integ="langevin", steps=100), members=6),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "traj", "host", "forces", "pairs", "rebuild", "batch", "serve"])
    if kind == "batch":
        return _unnamed(dict(_case("", "batch", 0, 0.0334, rc=9.0, integ="langevin",
                                   steps=2 * rng.randint(1, 5)), members=log_int(2, 48)))
    if kind == "serve":
        return _unnamed(dict(_case("", "serve", 0, 0.0334, rc=9.0, integ="langevin", steps=50), members=rng.randint(1, 3)))
    most = {"step": 72000, "traj": 30000, "host": 30000, "forces": 24000, "pairs": 8000, "rebuild": 1500}[kind]
    n = log_int(512, most)
    res = 0 if kind == "host" or rng.random() < 0.4 else rng.randint(3, 11)
    rho = rng.choice([0.0334, 0.0334, 0.03, 0.0255])
    rc = rng.choice([9.0, 10.0])
    # cells of 512 to 1100 waters: n of them in a box that need not be a cube
    cells = max(1, int(round(n / rng.uniform(650, 1000))))
    tx = max(1, int(round(cells ** (1.0 / 3.0))))
    ty = max(1, int(round(math.sqrt(cells / tx))))
    tz = max(1, int(round(cells / (tx * ty))))
    per = min(1100, max(512, int(round(n / (tx * ty * tz)))))
    integ = "nve" if kind == "host" else rng.choice(["langevin", "csvr", "csvr"])
    c = _case("", kind, per, rho, residues=res, tiles=(tx, ty, tz), drop=rng.randint(0, per // 9), rc=rc, integ=integ,
              steps=1 if kind == "host" else 20 if kind == "traj" else rng.randint(5, 20 if n < 40000 else 10),
              salt=0.15 if res and rng.random() < 0.3 else 0.0, corrected=kind == "forces" or rng.random() < 0.2,
              barostat=kind == "step" and integ == "csvr" and rng.random() < 0.4)
    if kind == "step" and res and n < 8000 and rng.random() < 0.3:
        c["lam"] = round(rng.uniform(0.0, 1.0), 2)
    if kind == "host":
        c["corrected"] = False
    return _unnamed(c)


def _unnamed(c):
    c.pop("name")
    return c


# ---------------------------------------------------------------------------
# constants of the OPC water model (float32 values, as the engine holds them)
# ---------------------------------------------------------------------------
_F = np.float32
_MO, _MH = 16.0, float(_F(1.008))
_MT = float(_F(16.0) + _F(2.0) * _F(1.008))
_Q_H = float(_F(0.6791) * _F(18.2223))
_Q_M = -2.0 * _Q_H
_O_SIGMA = float(_F(1.777167268) * (_F(2.0) / _F(1.122462048309373)))
_O_EPS = float(_F(0.2128008130))
_O_M = float(_F(0.15939833))
_C_H = float((_F(0.15939833) / _F(0.5395199719801114)) / _F(2.0))
_C_O = 1.0 - 2.0 * _C_H
_KCAL = float(_F(418.4))


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV).to(dtype)


def _sites(atom_pos, water):
    """(na + 4 nw, 3) float64 sites, atoms then O, H0, H1, M of each water;
    M rounded to float32 as it is held."""
    b = (water[:, 1] - water[:, 0]) + (water[:, 2] - water[:, 0])
    m = (water[:, 0] + b / b.norm(dim=1, keepdim=True) * _O_M).float().double()
    return torch.cat([atom_pos, torch.cat([water, m[:, None]], 1).reshape(-1, 3)])


def _tables(s, nw):
    """Charges, sigma, epsilon of the sites (epsilon 0: no LJ)."""
    one = torch.ones(nw, 1, dtype=torch.float64, device=DEV)
    w = lambda *v: (one * torch.tensor(v, dtype=torch.float64, device=DEV)).reshape(-1)  # noqa: E731
    return (torch.cat([_t(s["atom_q"]), w(0.0, _Q_H, _Q_H, _Q_M)]),
            torch.cat([_t(s["atom_sigma"]), w(_O_SIGMA, 0.0, 0.0, 0.0)]),
            torch.cat([_t(s["atom_eps"]), w(_O_EPS, 0.0, 0.0, 0.0)]))


def _pair_terms(d, q, sg, ep, rc, alpha):
    """Force over distance, energy and virial of pairs with displacement d."""
    r2 = (d * d).sum(-1)
    on = (r2 > 1e-12) & (r2 < rc * rc)
    r2 = torch.where(on, r2, torch.ones_like(r2))
    r = r2.sqrt()
    sr6 = (sg * sg / r2) ** 3
    ec = q * torch.erfc(alpha * r) / r
    f = (24.0 * ep * (2.0 * sr6 * sr6 - sr6) + ec
         + q * (2.0 * alpha / math.sqrt(math.pi)) * torch.exp(-(alpha * alpha) * r2)) / r2
    e = 4.0 * ep * (sr6 * sr6 - sr6) + ec
    f = torch.where(on, f, torch.zeros_like(f))
    return f, torch.where(on, e, torch.zeros_like(e)), f * r2


def _all_pairs(x, q, sg, ep, ext, rc, alpha, na, rows=None):
    """Sums over every ordered site pair within rc: forces (n, 3), and half
    the sums of energy, energy of pairs with an atom, and virial."""
    n = len(x)
    rows = rows or max(1, min(n, 20_000_000 // n))
    f = torch.empty_like(x)
    tot = torch.zeros(3, dtype=torch.float64, device=DEV)
    se = ep.sqrt()
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = x[a:b, None] - x[None]
        d = d - torch.round(d / ext) * ext
        fs, e, w = _pair_terms(d, q[a:b, None] * q[None], 0.5 * (sg[a:b, None] + sg[None]),
                               se[a:b, None] * se[None], rc, alpha)
        f[a:b] = (fs[..., None] * d).sum(1)
        water = e[max(0, na - a):, na:].sum() if b > na else 0.0
        tot += torch.stack([e.sum(), e.sum() - water, w.sum()])
    return f, 0.5 * tot


def _take_pairs(x, i, j, q, sg, ep, ext, rc, alpha, scale_lj, scale_q):
    """Forces, energy and virial of the given pairs, scaled."""
    d = x[i] - x[j]
    d = d - torch.round(d / ext) * ext
    fs, e, w = _pair_terms(d, scale_q * q[i] * q[j], 0.5 * (sg[i] + sg[j]), scale_lj * (ep[i] * ep[j]).sqrt(), rc, alpha)
    f = torch.zeros_like(x)
    f.index_put_((i,), fs[:, None] * d, accumulate=True)
    f.index_put_((j,), -fs[:, None] * d, accumulate=True)
    return f, e.sum(), w.sum()


def _water_pairs(na, nw):
    """The six site pairs inside each water."""
    base = na + 4 * torch.arange(nw, device=DEV)
    ab = [(a, b) for a in range(4) for b in range(a + 1, 4)]
    return torch.cat([base + a for a, _ in ab]), torch.cat([base + b for _, b in ab])


def _index(s, key, width):
    return _t(np.asarray(s.get(key, np.zeros((0, width))), np.int64).reshape(-1, width), torch.int64)


def _short(s, x, nw, rc, alpha):
    """Short-range forces, energy, energy of pairs with an atom, virial."""
    na = len(x) - 4 * nw
    ext = _t(np.asarray(s["box_hi"], _F) - np.asarray(s["box_lo"], _F))
    q, sg, ep = _tables(s, nw)
    f, (e, ea, w) = _all_pairs(x, q, sg, ep, ext, rc, alpha, na)
    for (i, j), lj, co, atoms in ((_water_pairs(na, nw), 1.0, 1.0, 0.0),
                                  (tuple(_index(s, "excl", 2).T), 1.0, 1.0, 1.0),
                                  (tuple(_index(s, "pair14", 2).T), 0.5, 1.0 - 1.0 / 1.2, 1.0)):
        if not len(i):
            continue
        g, de, dw = _take_pairs(x, i, j, q, sg, ep, ext, rc, alpha, lj, co)
        f, e, ea, w = f - g, e - de, ea - atoms * de, w - dw
    return f, e, ea, w


def _spme(x, q, lo, ext, grid, alpha):
    """Smooth PME, order 4: forces and energy with the self term."""
    K = torch.tensor(grid, dtype=torch.float64, device=DEV)
    fr = (x - lo) / ext
    u = (fr - torch.floor(fr)) * K
    base = torch.floor(u)
    w = u - base
    o = 1.0 - w
    th = torch.stack([o ** 3 / 6, (3 * w ** 3 - 6 * w ** 2 + 4) / 6, (-3 * w ** 3 + 3 * w ** 2 + 3 * w + 1) / 6,
                      w ** 3 / 6], -1)
    dth = torch.stack([-0.5 * o ** 2, 1.5 * w ** 2 - 2 * w, -1.5 * w ** 2 + w + 0.5, 0.5 * w ** 2], -1)
    idx = torch.remainder(base[..., None].long() - 3 + torch.arange(4, device=DEV), K.long()[:, None])
    flat = ((idx[:, 0, :, None, None] * grid[1] + idx[:, 1, None, :, None]) * grid[2] + idx[:, 2, None, None, :])
    outer = lambda a, b, c: a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]  # noqa: E731
    Q = torch.zeros(grid[0] * grid[1] * grid[2], dtype=torch.float64, device=DEV)
    Q.index_put_((flat.reshape(-1),), (q[:, None, None, None] * outer(th[:, 0], th[:, 1], th[:, 2])).reshape(-1),
                 accumulate=True)
    m, bm = [], []
    for a in range(3):
        k = torch.arange(grid[a], dtype=torch.float64, device=DEV)
        z = sum(c * torch.exp(2j * math.pi * k * t / grid[a]) for t, c in enumerate((1 / 6, 4 / 6, 1 / 6)))
        bm.append(1.0 / z.abs() ** 2)
        m.append(torch.where(k <= grid[a] // 2, k, k - grid[a]) / ext[a])
    m2 = m[0][:, None, None] ** 2 + m[1][None, :, None] ** 2 + m[2][None, None, :] ** 2
    m2[0, 0, 0] = 1.0
    G = torch.exp(-math.pi ** 2 * m2 / alpha ** 2) / (math.pi * ext.prod() * m2)
    G = G * bm[0][:, None, None] * bm[1][None, :, None] * bm[2][None, None, :]
    G[0, 0, 0] = 0.0
    S = torch.fft.fftn(Q.reshape(tuple(grid)))
    e = 0.5 * (G * S.abs() ** 2).sum() - alpha / math.sqrt(math.pi) * (q * q).sum()
    phi = (torch.fft.ifftn(G * S).real * Q.numel()).reshape(-1)[flat]
    f = torch.stack([(outer(dth[:, 0], th[:, 1], th[:, 2]) * phi).sum((1, 2, 3)),
                     (outer(th[:, 0], dth[:, 1], th[:, 2]) * phi).sum((1, 2, 3)),
                     (outer(th[:, 0], th[:, 1], dth[:, 2]) * phi).sum((1, 2, 3))], 1)
    return -q[:, None] * K / ext * f, e


def _charged_spme(s, x, nw, grid, alpha):
    q, _, _ = _tables(s, nw)
    lo, hi = _t(s["box_lo"]), np.asarray(s["box_hi"], _F)
    ext = _t(hi - np.asarray(s["box_lo"], _F))
    on = q != 0
    f = torch.zeros_like(x)
    f[on], e = _spme(x[on], q[on], lo, ext, grid, alpha)
    return f, e


def _corrections(s, x, nw, alpha):
    """Removes erf(alpha r) q q / r of the excluded pairs."""
    na = len(x) - 4 * nw
    ext = _t(np.asarray(s["box_hi"], _F) - np.asarray(s["box_lo"], _F))
    q, _, _ = _tables(s, nw)
    f, e = torch.zeros_like(x), 0.0
    for (i, j), sc in ((_water_pairs(na, nw), 1.0), (tuple(_index(s, "excl", 2).T), 1.0),
                       (tuple(_index(s, "pair14", 2).T), 1.0 - 1.0 / 1.2)):
        if not len(i):
            continue
        d = x[i] - x[j]
        d = d - torch.round(d / ext) * ext
        r = d.norm(dim=1)
        qq = sc * q[i] * q[j]
        er = torch.erf(alpha * r)
        fs = -qq * (er / r ** 2 - 2 * alpha / math.sqrt(math.pi) * torch.exp(-(alpha * r) ** 2) / r) / r
        f.index_put_((i,), fs[:, None] * d, accumulate=True)
        f.index_put_((j,), -fs[:, None] * d, accumulate=True)
        e = e - (qq * er / r).sum()
    return f, e


def _bonded(s, p, ext):
    """Bonds, angles and dihedrals: forces and energy."""
    if not len(s.get("bonds", ())):
        return torch.zeros_like(p), 0.0
    p = p.detach().requires_grad_(True)
    mi = lambda d: d - torch.round(d.detach() / ext) * ext  # noqa: E731
    i, j = _index(s, "bonds", 2).T
    e = (_t(s["bond_k"]) * (mi(p[j] - p[i]).norm(dim=1) - _t(s["bond_r0"])) ** 2).sum()
    a, b, c = _index(s, "angles", 3).T
    u, v = mi(p[a] - p[b]), mi(p[c] - p[b])
    th = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
    e = e + (_t(s["angle_k"]) * (th - _t(s["angle_theta0"])) ** 2).sum()
    a, b, c, d = _index(s, "dihedrals", 4).T
    b1, b2, b3 = mi(p[b] - p[a]), mi(p[c] - p[b]), mi(p[d] - p[c])
    n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
    phi = torch.atan2((torch.linalg.cross(n1, n2) * b2).sum(1) / b2.norm(dim=1), (n1 * n2).sum(1))
    e = e + (_t(s["dihedral_k"]) * (1 + torch.cos(_t(s["dihedral_n"]) * phi - _t(s["dihedral_phase"])))).sum()
    return -torch.autograd.grad(e, p)[0], e.detach()


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------

def _turn(v, w):
    """v (n, k, 3) turned by the rotation vectors w (n, 3)."""
    t = w.norm(dim=1)[:, None, None]
    n = (w / w.norm(dim=1, keepdim=True).clamp_min(1e-12))[:, None].expand_as(v)
    return v * torch.cos(t) + torch.linalg.cross(n, v) * torch.sin(t) + n * (n * v).sum(-1, keepdim=True) * (1 - torch.cos(t))


@functools.lru_cache(maxsize=None)
def _cell(waters, rho, residues, salt):
    """A relaxed periodic unit cell: capped steepest descent of rigid waters
    and atoms on the short-range and bonded energy, in float64 and in an
    order of sums that does not vary."""
    box = float((waters / rho) ** (1.0 / 3.0))
    if residues:
        s, _ = peptide.solvated_system(box, waters, n_res=(residues,), seed=waters + 7 * residues, nacl_molar=salt)
    else:
        s = synth.water_box(waters, box, seed=waters)
    w = _t(s["water_pos"])
    p = _t(s["atom_pos"]).reshape(-1, 3)
    nw, na = len(w), len(p)
    ext = _t(np.asarray(s["box_hi"], _F))
    q, sg, ep = _tables(s, nw)
    skip = [(i, j) for i, j in (_water_pairs(na, nw), tuple(_index(s, "excl", 2).T), tuple(_index(s, "pair14", 2).T))]
    i, j = (torch.cat([k[a] for k in skip]) for a in (0, 1))
    rc = min(10.0, 0.5 * box)
    mass = torch.tensor([_MO, _MH, _MH], dtype=torch.float64, device=DEV)[None, :, None]
    n_it = 240
    for it in range(n_it):
        x = _sites(p, w)
        f, _ = _all_pairs(x, q, sg, ep, ext, rc, 0.26, na)
        g, _, _ = _take_pairs(x, i, j, q, sg, ep, ext, rc, 0.26, 1.0, 1.0)
        f = f - g
        cap = 1.0 - 0.8 * it / n_it
        if na:
            fa = f[:na] + _bonded(s, p, ext)[0]
            step = 4e-4 * fa
            p = p + step * (0.04 * cap / step.norm(dim=1, keepdim=True).clamp_min(0.04 * cap))
        fw = f[na:].reshape(nw, 4, 3)
        com = (w * mass).sum(1) / _MT
        r = x[na:].reshape(nw, 4, 3) - com[:, None]
        step = 2e-3 * fw.sum(1)
        step = step * (0.06 * cap / step.norm(dim=1, keepdim=True).clamp_min(0.06 * cap))
        rot = 8e-3 * torch.linalg.cross(r, fw).sum(1)
        rot = rot * (0.15 * cap / rot.norm(dim=1, keepdim=True).clamp_min(0.15 * cap))
        w = com[:, None] + step[:, None] + _turn(w - com[:, None], rot)
    out = dict(s)
    out["water_pos"], out["atom_pos"] = w.cpu().numpy(), p.cpu().numpy()
    return out, box


_PER_ATOM = ("atom_mass", "atom_q", "atom_sigma", "atom_eps", "bond_k", "bond_r0", "angle_k", "angle_theta0",
             "dihedral_k", "dihedral_n", "dihedral_phase", "constraint_r0")
_INDEXED = ("bonds", "angles", "dihedrals", "excl", "pair14", "constraints")


def _system(case, seed):
    """The case's system for a seed: tiled, thermally displaced, shifted
    through the periodic box, its waters in a random order."""
    cell, box = _cell(case["waters"], case["rho"], case["residues"], case["salt"])
    rng = np.random.default_rng([seed, case["waters"], case["residues"], case["drop"]])
    tiles = np.array([case["tx"], case["ty"], case["tz"]])
    ext = (box * tiles).astype(_F)
    off = np.stack(np.meshgrid(*[np.arange(t) for t in tiles], indexing="ij"), -1).reshape(-1, 3) * box
    n = len(off)
    w = (cell["water_pos"][None] + off[:, None, None]).reshape(-1, 3, 3)
    w = w[np.sort(rng.permutation(len(w))[case["drop"]:])][rng.permutation(len(w) - case["drop"])]
    s = {"box_lo": np.zeros(3, _F), "box_hi": ext}
    # thermal displacement: molecules by 0.07 A, turned by 0.1 rad per axis
    com = (w[:, :1] * _MO + w[:, 1:2] * _MH + w[:, 2:] * _MH) / _MT
    turned = _turn(torch.from_numpy(w - com), torch.from_numpy(rng.normal(scale=0.1, size=(len(w), 3)))).numpy()
    shift = rng.uniform(0.0, 1.0, 3) * ext
    w = com + turned + rng.normal(scale=0.07, size=(len(w), 1, 3)) + shift
    w = w - np.floor(w[:, :1] / ext) * ext
    o, h = w[:, :1], w[:, 1:] - w[:, :1]
    s["water_pos"] = np.concatenate([o, o + h], 1).astype(_F)
    na = len(cell["atom_pos"])
    p = (cell["atom_pos"][None] + off[:, None]).reshape(-1, 3) + shift
    for k in _PER_ATOM:
        if len(cell.get(k, ())):
            s[k] = np.tile(np.asarray(cell[k], _F), n)
        elif k.startswith("atom_"):
            s[k] = np.zeros(0, _F)
    for k in _INDEXED:
        if len(cell.get(k, ())):
            a = np.asarray(cell[k], np.int64)
            s[k] = (a[None] + (np.arange(n) * na)[:, None, None]).reshape(-1, a.shape[1]).astype(np.uint32)
    # a hydrogen moves with its heavy atom
    move = rng.normal(scale=0.03, size=(len(p), 3))
    if "constraints" in s:
        c = s["constraints"].astype(np.int64)
        move[c[:, 1]] = move[c[:, 0]]
    s["atom_pos"] = (p + move).astype(_F)
    s["water_vel"] = synth.rigid_mb_velocities(s["water_pos"].astype(np.float64), TEMP, rng)
    kt = float(synth.KB_NATIVE) * TEMP
    s["atom_vel"] = rng.normal(size=s["atom_pos"].shape) * np.sqrt(kt / np.maximum(s["atom_mass"], 1e-6))[:, None]
    synth.remove_com_and_scale(s, TEMP, 6 * len(w) + 3 * len(p) - len(s.get("constraints", ())) - 3)
    s["water_vel"], s["atom_vel"] = s["water_vel"].astype(_F), s["atom_vel"].astype(_F)
    grid = tuple(synth.fft_size(int(math.ceil(e - 1e-3))) for e in ext)
    return s, grid


def _config(case, system, grid, seed):
    integ = {"langevin": md.LangevinMiddle(gamma=10.0), "csvr": md.VerletVelocity(thermostat=0.1),
             "nve": md.VerletVelocity(thermostat=None)}[case["integ"]]
    cfg = md.MdConfig(integrator=integ, coulomb_cutoff=case["rc"], lj_cutoff=case["rc"],
                      spme_alpha=synth.ewald_alpha(case["rc"]), spme_grid=grid, seed=seed,
                      spme_interval=case["spme_every"], ewald_corrections=case["corrected"],
                      full_energy=case["corrected"], rattle_velocities=case["rattle"])
    if case["barostat"]:
        cfg.barostat_cfg = md.BarostatCfg(pressure_target=1.0, tau=5.0, solvent_compressibility=4.5e-5)
    if case["lam"] >= 0.0:
        # the atoms of the first cell's peptide (its ions come after them)
        cell, _ = _cell(case["waters"], case["rho"], case["residues"], case["salt"])
        cfg.alch_range, cfg.alch_lambda = (0, int(np.asarray(cell["bonds"]).max()) + 1), case["lam"]
    return cfg


def _members(case, seed):
    """Members of 512 to 8000 waters: cells of five sizes, some with a
    peptide, in 1 to 8 copies, each with some waters taken out."""
    out = []
    for k in range(case["members"]):
        waters, res = ((512, 0), (640, 10), (760, 0), (880, 10), (1000, 0))[k % 5]
        tiles = ((1, 1, 1), (2, 1, 1), (2, 2, 1), (1, 1, 2), (2, 2, 2), (1, 1, 1), (3, 1, 1))[k % 7]
        c = dict(case, waters=waters, residues=res, tx=tiles[0], ty=tiles[1], tz=tiles[2], drop=(11 * k) % 60)
        s, grid = _system(c, 1000 * seed + k)
        out.append((s, _config(c, s, grid, 1000 * seed + k)))
    return out


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def _buffers(s):
    na, nw = len(s["atom_pos"]), len(s["water_pos"])
    return {"atom_pos": _pinned(na, 3), "atom_vel": _pinned(na, 3), "water_pos": _pinned(nw, 3, 3),
            "water_vel": _pinned(nw, 3, 3)}


def _water_sites(s):
    w = np.asarray(s["water_pos"], np.float64)
    b = (w[:, 1] - w[:, 0]) + (w[:, 2] - w[:, 0])
    m = w[:, 0] + b / np.linalg.norm(b, axis=1, keepdims=True) * _O_M
    return [np.ascontiguousarray(a, _F) for a in (w[:, 0], m, w[:, 1], w[:, 2])]


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        members = _members(case, seed)
        b = md.MdBatch([s for s, _ in members], [c for _, c in members])
        return {"kind": kind, "batch": b, "steps": case["steps"], "out": _pinned(int(b.state_layout()[-1]))}
    if kind == "serve":
        return {"kind": kind, "members": _members(case, seed), "steps": case["steps"]}
    s, grid = _system(case, seed)
    if kind in ("pairs", "rebuild"):
        f = gpu_interface.ForcesPositsGpu(len(s["atom_pos"]), len(s["water_pos"]), case["rc"],
                                          synth.ewald_alpha(case["rc"]), case["rc"])
        st = {"kind": kind, "forces": f, "system": s, "water": _water_sites(s), "pairs": None,
              "extent": (s["box_hi"] - s["box_lo"]).astype(_F)}
        if kind == "pairs":
            st["pairs"] = _build_list(st)
        return st
    sim = md.MdState(s, _config(case, s, grid, seed))
    st = {"kind": kind, "sim": sim, "steps": case["steps"]}
    if kind == "traj":
        sim.enable_snapshots(10, capacity=max(1, case["steps"] // 10), velocities=True)
    elif kind in ("step", "host"):
        st["out"] = _buffers(s)
        if kind == "host":
            for k, v in st["out"].items():
                v[...] = s[k]
    return st


def _build_list(st):
    s = st["system"]
    return gpu_interface.PerNeighborGpu.build(
        st["forces"], s["atom_pos"], st["water"][0], s["atom_q"], s["atom_sigma"], s["atom_eps"], s["box_lo"],
        s["box_hi"], SKIN, excl=s.get("excl"), pair14=s.get("pair14"))


_SCALARS = ("potential", "kinetic", "temperature")


def run(state):
    kind = state["kind"]
    if kind in ("step", "host"):
        out = state["out"]
        e = state["sim"].step_host(DT, state["steps"], out if kind == "host" else {}, out)
        return dict(out, **{k: e[k] for k in _SCALARS})
    if kind == "traj":
        state["sim"].step(DT, state["steps"])
        return [{k: f[k] for k in ("pos", "vel") + _SCALARS} for f in state["sim"].read_snapshots()]
    if kind == "forces":
        r = state["sim"].forces()
        return {k: r[k] for k in ("f_atoms", "f_water", "potential", "virial")}
    if kind in ("pairs", "rebuild"):
        if kind == "rebuild":
            state["pairs"] = _build_list(state)
        fd, fw, w, e = gpu_interface.force_nonbonded_gpu(state["forces"], state["pairs"], state["system"]["atom_pos"],
                                                         state["water"], state["extent"])
        return {"f_dyn": fd, "f_water": fw, "virial": w, "energy": e}
    if kind == "batch":
        e = state["batch"].step_host(DT, state["steps"], None, state["out"], energies=True)
        return dict({k: np.array([m[k] for m in e]) for k in _SCALARS}, state=state["out"])
    # requests of one to three rounds of 50 steps, all waiting at the start
    reqs = [serve.Request(rid=k, system=s, cfg=c, n_steps=50 * (1 + (k * state["steps"] // 50) % 3), arrival=0.0)
            for k, (s, c) in enumerate(state["members"])]
    serve.Server(max_members=4, round_steps=50, dt=DT).run(reqs)
    return [dict({k: r.state[k] for k in ("atom_pos", "atom_vel", "water_pos", "water_vel")},
                 potential=r.energies["potential"]) for r in reqs]


# ---------------------------------------------------------------------------
# work, tolerance and the float64 answers
# ---------------------------------------------------------------------------

def _member_sizes(case):
    for k in range(case["members"]):
        waters, res = ((512, 0), (640, 10), (760, 0), (880, 10), (1000, 0))[k % 5]
        copies = (1, 2, 4, 2, 8, 1, 3)[k % 7]
        yield waters * copies, 17 * res * copies, waters * copies / case["rho"]


def _evaluation(nw, na, vol, rc):
    """Operations of the pairs inside the cutoff (19 for the distance, 15
    for LJ, 23 for screened Coulomb) and of the mesh (64 stencil points per
    charge each way, two transforms)."""
    shell = 4.0 / 3.0 * math.pi * rc ** 3 / vol / 2.0
    lj, co = (nw + na) ** 2 * shell, (3 * nw + na) ** 2 * shell
    nq = 3 * nw + na
    mesh = nq * 64 * 8.0 + 5.0 * vol * math.log2(vol)
    return lj * 34.0 + co * 42.0, mesh


def work(case):
    if case["kind"] in ("batch", "serve"):
        sizes = list(_member_sizes(case))
    else:
        copies = case["tx"] * case["ty"] * case["tz"]
        sizes = [(case["waters"] * copies - case["drop"], 17 * case["residues"] * copies,
                  case["waters"] * copies / case["rho"])]
    kind, steps = case["kind"], case["steps"] if case["kind"] in ("step", "traj", "host", "batch", "serve") else 1
    bytes_, flops = 0.0, 0.0
    for nw, na, vol in sizes:
        pf, mf = _evaluation(nw, na, vol, case["rc"])
        # positions and velocities in and out; or positions in, float64 forces out
        bytes_ += 144.0 * nw + 48.0 * na if kind not in ("forces", "pairs", "rebuild") else 36.0 * (4 * nw + na)
        if kind in ("pairs", "rebuild"):
            flops += pf
            if kind == "pairs":  # the installed list is an input: 20 bytes a pair
                bytes_ += 20.0 * 10 * nw ** 2 / 2 / vol * 4 / 3 * math.pi * (case["rc"] + SKIN) ** 3
            continue
        mesh = (1.0 if kind == "forces" else 1.0 / case["spme_every"]) * (3.0 if case["lam"] >= 0.0 else 1.0)
        flops += steps * (pf + mesh * mf)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Four times the largest difference seen over two passes (or, for single
    evaluations, from the float64 answer) when the float sums are grouped
    otherwise: other work-item lengths, list buffers and chunk sizes.
    Velocities set it; a step's rounding grows along the trajectory."""
    return {"step": {"rel": 2e-3, "max": 2.5e-2}, "traj": {"rel": 2e-3, "max": 2.5e-2},
            "serve": {"rel": 8e-3, "max": 0.32}, "batch": {"rel": 2e-5, "max": 2e-3},
            "host": {"rel": 3e-5, "max": 1e-3}, "forces": {"rel": 8e-6, "max": 4e-4},
            "pairs": {"rel": 3e-5, "max": 1e-3}, "rebuild": {"rel": 3e-5, "max": 1e-3}}[case["kind"]]


def _exact_forces(case, seed):
    s, grid = _system(case, seed)
    nw, alpha = len(s["water_pos"]), float(_F(synth.ewald_alpha(case["rc"])))
    x = _sites(_t(s["atom_pos"]), _t(s["water_pos"]))
    na = len(x) - 4 * nw
    f, e, _, _ = _short(s, x, nw, case["rc"], alpha)
    for g, de in (_charged_spme(s, x, nw, grid, alpha), _corrections(s, x, nw, alpha)):
        f, e = f + g, e + de
    fb, eb = _bonded(s, x[:na], _t(s["box_hi"]))
    f[:na] += fb
    return {"f_atoms": f[:na], "f_water": f[na:].reshape(nw, 4, 3), "potential": float(e + eb), "virial": None}


def _exact_pairs(case, seed):
    s, _ = _system(case, seed)
    nw, alpha = len(s["water_pos"]), float(_F(synth.ewald_alpha(case["rc"])))
    x = _sites(_t(s["atom_pos"]), _t(s["water_pos"]))
    na = len(x) - 4 * nw
    f, _, ea, w = _short(s, x, nw, case["rc"], alpha)
    fw = f[na:].reshape(nw, 4, 3)
    return {"f_dyn": f[:na], "f_water": {1: fw[:, 0], 2: fw[:, 3], 3: fw[:, 1], 4: fw[:, 2]},
            "virial": float(w), "energy": float(ea)}


def _exact_host_step(case, seed):
    """One velocity-Verlet step of rigid waters: half kick, drift (centre of
    mass and a rotation at the angular velocity of the kicked sites), half
    kick."""
    s, grid = _system(case, seed)
    alpha = float(_F(synth.ewald_alpha(case["rc"])))
    ext = _t(s["box_hi"])
    w, v = _t(s["water_pos"]), _t(s["water_vel"])
    nw = len(w)
    mass = torch.tensor([_MO, _MH, _MH], dtype=torch.float64, device=DEV)[None, :, None]
    none = torch.zeros(0, 3, dtype=torch.float64, device=DEV)

    def accel(w):
        x = _sites(none, w)
        f, _, _, _ = _short(s, x, nw, case["rc"], alpha)
        g, e = _charged_spme(s, x, nw, grid, alpha)
        f = (f + g).reshape(nw, 4, 3)
        f = f[:, :3] + f[:, 3:] * torch.tensor([_C_O, _C_H, _C_H], dtype=torch.float64, device=DEV)[None, :, None]
        return f * _KCAL / mass, e

    v = v + 0.5 * DT * accel(w)[0]
    com, vc = (w * mass).sum(1) / _MT, (v * mass).sum(1) / _MT
    r, u = w - com[:, None], v - vc[:, None]
    L = (torch.linalg.cross(r, u) * mass).sum(1)
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    inertia = (mass[..., None] * ((r * r).sum(-1)[..., None, None] * eye - r[..., :, None] * r[..., None, :])).sum(1)
    om = torch.linalg.solve(inertia, L[..., None])[..., 0]
    r = _turn(r, om * DT)
    w = com[:, None] + DT * vc[:, None] + r
    w = w - torch.floor(w[:, :1] / ext) * ext
    v = vc[:, None] + torch.linalg.cross(om[:, None].expand_as(r), r)
    a, e = accel(w.float().double())
    v = v + 0.5 * DT * a
    return {"atom_pos": None, "atom_vel": None, "water_pos": w, "water_vel": v, "potential": float(e),
            "kinetic": float(0.5 * (mass * v * v).sum() / _KCAL), "temperature": None}


def exact(case, seed):
    """None for runs of many steps: their thermostats draw random numbers,
    and rounding grows along a trajectory."""
    fn = {"forces": _exact_forces, "pairs": _exact_pairs, "rebuild": _exact_pairs, "host": _exact_host_step}.get(case["kind"])
    return fn(case, seed) if fn else None
