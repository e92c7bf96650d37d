"""The work a user of this library has it do, as cases that can be timed and compared.

Kinds of a case:

step     one MD step of the plain path between two list rebuilds, as SPONGE's
         loop runs it: the conditional list update, then the LJ + PME direct
         force (``PlainPath.step``).  ``terms``: "f" forces, the step between
         energy outputs; "totals" forces and the FP64 energy and virial
         totals; "fev" forces with per-atom energies and virials.  The atoms
         move between the calls as they do between the steps of a run, so the
         pruned lists are redone about every third step.  ``fused``: the PME
         excluded-pair correction in the same call.
rebuild  the step on which the list is rebuilt: forced update and force;
         ``full_list`` also makes the full list that many-body modules read.
soft     one step of an alchemical run through LJ_SOFT_CORE.
batch    independent systems stepped together (leap-frog, SETTLE, thermostat,
         list rebuilds every 20 steps) from captured graphs, their energies
         and final state read back: the equilibration of freshly built boxes.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sponge2.0_b200"))

from spgnb import systems as S  # noqa: E402
from spgnb.batch import Batch  # noqa: E402
from spgnb.engine import PlainPath, SoftCorePath  # noqa: E402

DENSITY = 0.0334     # molecules (waters and solutes) per cubic Angstrom
SKIN = 2.0
PERTURBED = 40       # atoms of the alchemical cases' ligand
FULL_LIST_MAX = 1200
# displacements of successive steps, in units of the largest: a run moves on
# and the pruned lists (redone past 0.5 A) follow
AMPLITUDES = (0.0, 0.2, 0.4, 0.55, 0.4, 0.2)
NO_REBUILD = 1 << 28


def _step(name, waters, solutes, cutoff, terms, **kw):
    return dict(kind="step", name=name, waters=waters, solutes=solutes, cutoff=cutoff, terms=terms,
                triclinic=kw.get("triclinic", False), fused=kw.get("fused", False))


def listed():
    return [
        # small peptide-in-water sizes, where latency and launches count
        _step("water1944_f", 648, 0, 8.0, "f"),
        # the 40 A water box, between and on energy outputs
        _step("water6480_f", 2160, 0, 10.0, "f"),
        _step("water6480_fev", 2160, 0, 10.0, "fev"),
        # a skewed cell at constant pressure: energy and virial totals
        _step("triclinic5500_totals", 1800, 100, 8.0, "totals", triclinic=True),
        # a solvated protein's size, an odd atom count, PME's correction fused
        _step("mixed24k_f_fused", 7411, 1780, 9.0, "f", fused=True),
        # the 96,000-atom mixed box: the common production size
        _step("mixed96k_f", 30000, 6000, 10.0, "f"),
        _step("mixed96k_fev", 30000, 6000, 10.0, "fev"),
        # the 1.0 M-atom box, rc 12
        _step("water1m_f", 333333, 0, 12.0, "f"),
        # rebuild steps: a small box with a many-body module's full list, the 96k box
        dict(kind="rebuild", name="rebuild8200_full_list", waters=2600, solutes=400, cutoff=8.0, full_list=True),
        dict(kind="rebuild", name="rebuild96k", waters=30000, solutes=6000, cutoff=10.0, full_list=False),
        # free-energy run of a solvated ligand
        dict(kind="soft", name="soft19k_f", waters=6000, solutes=1200, cutoff=9.0, terms="f", lam=0.6),
        # 20 uneven systems of 1,500-24,000 atoms, one refresh interval
        dict(kind="batch", name="batch20", systems=20, n_min=1500, n_max=24000, steps=20),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("step", "rebuild", "soft", "batch"), (6, 2, 1, 1))[0]
    if kind == "batch":
        return dict(kind="batch", systems=_log_uniform(rng, 1, 20), n_min=1500, n_max=_log_uniform(rng, 3000, 24000),
                    steps=20)
    molecules = _log_uniform(rng, 700 if kind != "soft" else 2500, 36000)
    solutes = int(molecules * rng.choice((0.0, rng.uniform(0.0, 0.15), 0.2)))
    if kind == "soft":
        solutes = max(solutes, 4 * PERTURBED)
    half = 0.5 * (molecules / DENSITY) ** (1.0 / 3.0)
    cutoff = rng.choice([rc for rc in (8.0, 9.0, 10.0, 12.0) if rc + SKIN <= half])
    c = dict(kind=kind, waters=molecules - solutes, solutes=solutes, cutoff=cutoff)
    if kind == "rebuild":
        c["full_list"] = rng.random() < 0.3
    elif kind == "soft":
        c["terms"] = rng.choice(("f", "totals"))
        c["lam"] = round(rng.uniform(0.1, 0.9), 3)
    else:
        c["terms"] = rng.choice(("f", "f", "totals", "fev"))
        c["triclinic"] = rng.random() < 0.15
        c["fused"] = rng.random() < 0.3
    return c


# ------------------------------------------------------------------ inputs
def _box(case):
    molecules = case["waters"] + case["solutes"]
    L = (molecules / DENSITY) ** (1.0 / 3.0)
    if case.get("triclinic"):
        # the same density in a cell skewed as the test systems' one is
        angles = (75.0, 80.0, 70.0)
        cell, _ = S.cell_from_box(1.0, 1.0, 1.0, *angles)
        L = (molecules / DENSITY / float(cell[0] * cell[2] * cell[5])) ** (1.0 / 3.0)
        return (0.97 * L, L, L / 0.97), angles
    return (L, L, L), (90.0, 90.0, 90.0)


def _system(case, seed):
    box, angles = _box(case)
    # a placement that cannot keep the solutes apart is drawn again
    for k in range(20):
        try:
            return S.water_system(case["waters"], box, 20 * seed + k, n_solute=case["solutes"],
                                  cutoff=case["cutoff"], skin=SKIN, angles=angles)
        except RuntimeError:
            if k == 19:
                raise


def _fep(case, seed):
    return S.fep_system(_system(case, seed), n_perturbed=PERTURBED, seed=seed % 100003, lam=case["lam"])


def _batch_systems(case, seed):
    # the library's uneven batch, the atom counts spread evenly over their
    # logarithm so that batches of different seeds cost the same
    rng = np.random.default_rng(seed)
    types = S.shared_solute_types()
    out = []
    for k in range(case["systems"]):
        x = (k + 0.5) / case["systems"]
        n_atoms = int(case["n_min"] * (case["n_max"] / case["n_min"]) ** x)
        rc = (8.0, 10.0, 12.0)[k % 3]
        n_sol = int(n_atoms * 0.15 * ((k * 7) % 11) / 10.0)
        n_w = (n_atoms - n_sol) // 3
        L = ((n_w + n_sol) / DENSITY) ** (1.0 / 3.0)
        rc = max(v for v in (8.0, 10.0, 12.0) if v <= rc and (v + SKIN <= 0.5 * L or v == 8.0))
        for attempt in range(20):
            try:
                out.append(S.water_system(n_w, L, int(rng.integers(1 << 31)), n_solute=n_sol, cutoff=rc, skin=SKIN,
                                          solute_types=types))
                break
            except RuntimeError:
                if attempt == 19:
                    raise
    return out


def _moves(n, seed):
    """Directions and lengths (at most 1) of the atoms' displacements."""
    rng = np.random.default_rng(seed + 77)
    u = rng.normal(size=(n, 3))
    u *= (rng.uniform(0.0, 1.0, n) / np.linalg.norm(u, axis=1))[:, None]
    return u


def _frames(s, seed):
    u = _moves(s.n, seed)
    return [torch.from_numpy((s.crd + a * u).astype(np.float32)).cuda() for a in AMPLITUDES]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "k": 0}
    if kind == "step":
        s = _system(case, seed)
        st["path"] = p = PlainPath(s, refresh_interval=NO_REBUILD)
        if case["fused"]:
            p.lj.Fuse_PME_Excluded(s.n, p.excl_start, p.excl_list, p.excl_numbers, len(s.excl_list))
        st["frames"] = _frames(s, seed)
    elif kind == "rebuild":
        s = _system(case, seed)
        st["path"] = p = PlainPath(s, refresh_interval=NO_REBUILD)
        st["frames"] = _frames(s, seed)
        if case["full_list"]:
            counts, temp, overflow = p.nl.build_full(p.n, st["frames"][0], p.cell, p.rcell, 0.0, FULL_LIST_MAX)
            st["full"] = p.nl._full_out
    elif kind == "soft":
        fep = _fep(case, seed)
        st["path"] = SoftCorePath(fep, refresh_interval=NO_REBUILD)
        st["frames"] = _frames(st["path"].system, seed)
    else:
        st["batch"] = Batch(_batch_systems(case, seed), refresh_interval=20, thermostat_tau=0.01, temperature=300.0)
    return st


# --------------------------------------------------------------------- run
def _joined(energies, states):
    """A batch's energies and its systems' final states, one after another."""
    crd, vel, frc = (np.concatenate(a) for a in zip(*states))
    return {"energies": energies, "crd": crd, "vel": vel, "frc": frc}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        b = st["batch"]
        b.run(case["steps"], energy_interval=case["steps"])
        return _joined(b.energies(), [b.download(k) for k in range(b.n_ids)])
    p = st["path"]
    frame = st["frames"][st["k"] % len(AMPLITUDES)]
    st["k"] += 1
    if kind == "rebuild":
        p.update(0, forced=True, crd=frame)
        out = {"frc": p.force(crd=frame)}
        if case["full_list"]:
            counts, lists, overflow = p.nl.build_full(p.n, frame, p.cell, p.rcell, 0.0, FULL_LIST_MAX, out=st["full"])
            out.update(counts=counts, lists=lists, overflow=overflow)
        return out
    terms = case["terms"]
    energy = terms != "f"
    out = {"frc": p.step(1, need_energy=energy, need_virial=energy, crd=frame, per_atom=terms == "fev")}
    if terms == "fev":
        out.update(energy=p.atom_energy, virial=p.atom_virial, direct=p.atom_direct)
    if energy:
        out["totals"] = p.lj.totals()
    return out


# -------------------------------------------------------------------- work
# operations of a pair: 45 for the force, 22 more for energy and virial; 9 for
# a distance test of the list
def _pairs(n, volume, radius):
    return 0.5 * n * min(n, n / volume * 4.0 / 3.0 * math.pi * radius ** 3)


def work(case):
    if case["kind"] == "batch":
        b = f = 0.0
        for k in range(case["systems"]):
            x = (k + 0.5) / case["systems"]
            n = int(case["n_min"] * (case["n_max"] / case["n_min"]) ** x)
            V = n / 0.1
            rc = (8.0, 10.0, 12.0)[k % 3]
            rc = max(v for v in (8.0, 10.0, 12.0) if v <= rc and (v + SKIN <= 0.5 * V ** (1.0 / 3.0) or v == 8.0))
            # a step reads and writes positions and velocities; one rebuild
            b += case["steps"] * n * (2 * 24 + 12)
            f += case["steps"] * 45 * _pairs(n, V, rc) + 9 * _pairs(n, V, rc + SKIN)
        return {"bytes": b, "flops": f}
    n = 3 * case["waters"] + case["solutes"]
    V = (case["waters"] + case["solutes"]) / DENSITY
    rc = case["cutoff"]
    inside = _pairs(n, V, rc)
    terms = case.get("terms", "f")
    # coordinates, charge and type in; the force out (and read: it is added to)
    b = n * (12 + 4 + 4 + 24)
    f = inside * 45
    if terms != "f":
        f += inside * 22
    if terms == "fev":
        b += n * 2 * (4 + 4 + 24)
    if case["kind"] == "rebuild":
        listed_pairs = _pairs(n, V, rc + SKIN)
        f += 9 * listed_pairs
        b += n * (12 + 8)
        if case["full_list"]:
            b += 2 * listed_pairs * 4
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    if case["kind"] == "batch":
        # the steps amplify the forces' rounding: 8e-5 from 64 bits after 20 of
        # them (velocities), about ten times that after the next 20
        return {"rel": 2e-3, "max": 0.5}
    # four times the distance from 64 bits: 8e-7 for forces and totals, 6e-6
    # for the per-atom energies, sums of cancelling terms
    return {"rel": 2.4e-5 if case.get("terms") == "fev" else 4e-6, "max": 1e-3}


# ------------------------------------------------------------------- exact
def _image(d, cell):
    """Minimum image (one rounding per box vector), lower-triangular cell."""
    a11, a21, a22, a31, a32, a33 = [float(v) for v in cell]
    sz = torch.floor(d[..., 2] / a33 + 0.5)
    y = d[..., 1] - sz * a32
    x = d[..., 0] - sz * a31
    z = d[..., 2] - sz * a33
    sy = torch.floor(y / a22 + 0.5)
    x = x - sy * a21
    y = y - sy * a22
    x = x - a11 * torch.floor(x / a11 + 0.5)
    return torch.stack((x, y, z), -1)


def _pair_list(x, cell, rc, mol):
    """All pairs i < j within rc (and not in one molecule), by tiles of the box."""
    n = x.shape[0]
    a11, a21, a22, a31, a32, a33 = [float(v) for v in cell]
    orth = a21 == a31 == a32 == 0.0
    nt = [int(a11 // rc), int(a22 // rc)] if orth and n > 20000 else [1, 1]
    if min(nt) < 4:
        nt = [1, 1]
    tx = torch.clamp((torch.remainder(x[:, 0] / a11, 1.0) * nt[0]).long(), max=nt[0] - 1)
    ty = torch.clamp((torch.remainder(x[:, 1] / a22, 1.0) * nt[1]).long(), max=nt[1] - 1)
    tile = tx * nt[1] + ty
    order = torch.argsort(tile, stable=True)
    start = torch.searchsorted(tile[order].contiguous(), torch.arange(nt[0] * nt[1] + 1, device=x.device)).tolist()
    members = [order[start[t]:start[t + 1]] for t in range(nt[0] * nt[1])]
    out = []
    for t in range(nt[0] * nt[1]):
        cx, cy = divmod(t, nt[1])
        near = sorted({((cx + dx) % nt[0]) * nt[1] + (cy + dy) % nt[1] for dx in (-1, 0, 1) for dy in (-1, 0, 1)})
        cand = torch.cat([members[u] for u in near])
        rows = max(1, int(1.5e8 // max(1, cand.numel())))
        for r0 in range(0, members[t].numel(), rows):
            own = members[t][r0:r0 + rows]
            d = _image(x[cand][None, :, :] - x[own][:, None, :], cell)
            ok = ((d * d).sum(-1) < rc * rc) & (own[:, None] < cand[None, :]) & (mol[own][:, None] != mol[cand][None, :])
            a, b = torch.nonzero(ok, as_tuple=True)
            out.append((own[a], cand[b]))
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _molecules(s):
    mol = np.arange(s.n)
    w = s.n - s.n_solute
    mol[s.n_solute:] = s.n_solute + np.arange(w) // 3
    return torch.from_numpy(mol).cuda()


def _tri(a, b):
    hi, lo = torch.maximum(a, b), torch.minimum(a, b)
    return hi * (hi + 1) // 2 + lo


def _sums(n, i, j, d, f, elj, ec, frc, e_lj, e_c, vir):
    g = f[:, None] * d
    frc.index_add_(0, i, g)
    frc.index_add_(0, j, -g)
    if elj is None:
        return
    e_lj.index_add_(0, i, elj)
    e_c.index_add_(0, i, ec)
    w = -torch.stack((g[:, 0] * d[:, 0], 2 * g[:, 0] * d[:, 1], g[:, 1] * d[:, 1], 2 * g[:, 0] * d[:, 2],
                      2 * g[:, 1] * d[:, 2], g[:, 2] * d[:, 2]), -1)
    vir.index_add_(0, i, w)


def _screened(beta, r, qq):
    """Screened Coulomb: (force / r, energy)."""
    e = qq * torch.erfc(beta * r) / r
    return e / (r * r) + qq * (2.0 / math.sqrt(math.pi)) * beta * torch.exp(-(beta * r) ** 2) / (r * r), e


def _plain_pairs(s, x, q, pairs=None):
    """64-bit forces and the owner's (lower index) energies and virials."""
    dev = x.device
    n = s.n
    frc = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    e_lj = torch.zeros(n, dtype=torch.float64, device=dev)
    e_c = torch.zeros_like(e_lj)
    vir = torch.zeros((n, 6), dtype=torch.float64, device=dev)
    A = torch.from_numpy(s.pair_A.astype(np.float64)).to(dev)
    B = torch.from_numpy(s.pair_B.astype(np.float64)).to(dev)
    t = torch.from_numpy(s.atom_type.astype(np.int64)).to(dev)
    I, J = _pair_list(x, s.cell, s.cutoff, _molecules(s)) if pairs is None else pairs
    step = 30_000_000
    for c in range(0, I.numel(), step):
        i, j = I[c:c + step], J[c:c + step]
        d = _image(x[j] - x[i], s.cell)
        r = d.norm(dim=-1)
        k = _tri(t[i], t[j])
        r6 = r ** -6
        fc, ec = _screened(s.beta, r, q[i] * q[j])
        f = (B[k] - A[k] * r6) * r6 / (r * r) - fc
        _sums(n, i, j, d, f, (A[k] / 12 * r6 - B[k] / 6) * r6, ec, frc, e_lj, e_c, vir)
    return frc, e_lj, e_c, vir


def _soft_pairs(fep, s, x, q):
    """The two-state pair of LJ_SOFT_CORE in 64 bits."""
    dev = x.device
    n = s.n
    frc = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    e_lj = torch.zeros(n, dtype=torch.float64, device=dev)
    e_c = torch.zeros_like(e_lj)
    vir = torch.zeros((n, 6), dtype=torch.float64, device=dev)
    up = lambda a: torch.from_numpy(a.astype(np.float64)).to(dev)  # noqa: E731
    tabs = [up(a) for a in (fep.AA, fep.AB, fep.BA, fep.BB)]
    ta = torch.from_numpy(fep.type_a.astype(np.int64)).to(dev)
    tb = torch.from_numpy(fep.type_b.astype(np.int64)).to(dev)
    I, J = _pair_list(x, s.cell, s.cutoff, _molecules(s))
    # the ligand's own exclusions
    gone = torch.from_numpy(np.repeat(np.arange(n), s.excl_numbers) * n + s.excl_list).to(dev)
    keep = ~torch.isin(I * n + J, gone)
    i, j = I[keep], J[keep]
    d = _image(x[j] - x[i], s.cell)
    r = d.norm(dim=-1)
    ka, kb = _tri(ta[i], ta[j]), _tri(tb[i], tb[j])
    AA, AB, BA, BB = tabs[0][ka], tabs[1][ka], tabs[2][kb], tabs[3][kb]
    qq = q[i] * q[j]
    l, l_ = fep.lam, 1.0 - fep.lam
    soft = ~((AA * BA != 0) | (AA + BA == 0))
    s6, s6min = fep.sigma ** 6, fep.sigma_min ** 6

    def sigma6(a, b):
        some = (a != 0) & (b != 0)
        return torch.where(some, torch.clamp(0.5 * a / torch.where(some, b, torch.ones_like(b)), min=s6min),
                           torch.full_like(a, s6))

    zero = torch.zeros_like(r)
    ra = (r ** 6 + torch.where(soft, fep.alpha * l ** fep.p * sigma6(AA, AB), zero)) ** (1.0 / 6.0)
    rb = (r ** 6 + torch.where(soft, fep.alpha * l_ ** fep.p * sigma6(BA, BB), zero)) ** (1.0 / 6.0)

    def state(A, B, rs):
        # dU/dr / r at the soft distance: the factor r^4 / rs^5 of drs/dr
        i6 = rs ** -6
        lj = (B - A * i6) * i6 * rs ** -2
        fc, ec = _screened(s.beta, rs, qq)
        chain = (r / rs) ** 4
        return (lj - fc) * chain, (A / 12 * i6 - B / 6) * i6, ec

    fa, ela, eca = state(AA, AB, ra)
    fb, elb, ecb = state(BA, BB, rb)
    _sums(n, i, j, d, l_ * fa + l * fb, l_ * ela + l * elb, l_ * eca + l * ecb, frc, e_lj, e_c, vir)
    return frc, e_lj, e_c, vir


def _excluded(s, x, q, frc, e, vir):
    """PME's excluded-pair correction added to forces, energies and virials."""
    i = torch.from_numpy(np.repeat(np.arange(s.n), s.excl_numbers)).cuda()
    j = torch.from_numpy(s.excl_list.astype(np.int64)).cuda()
    d = _image(x[j] - x[i], s.cell)
    r = d.norm(dim=-1)
    qq = q[i] * q[j]
    fc, ec = _screened(s.beta, r, qq)
    # erf / r = 1 / r - erfc / r, taken out
    f = qq / r ** 3 - fc
    zero = torch.zeros_like(e)
    _sums(s.n, i, j, d, f, -(qq / r - ec), torch.zeros_like(ec), frc, e, zero, vir)


def _exact_batch(case, seed):
    dt = 0.002 * float(np.float32(20.455))
    all_energies, states = [], []
    for s in _batch_systems(case, seed):
        x = torch.from_numpy(s.crd.astype(np.float64)).cuda()
        v = torch.from_numpy(s.vel.astype(np.float64)).cuda()
        q = torch.from_numpy(s.charge.astype(np.float64)).cuda()
        m = torch.from_numpy(s.mass.astype(np.float64)).cuda()[:, None]
        w0 = s.n_solute
        lam = 1.0
        kT0 = 0.00198716 * 300.0
        ndof = max(1, 3 * s.n - 3 * s.n_waters - 3)
        # distances of the rigid water and the weights of its constraints
        cons = ((0, 1, 0.9572 ** 2), (0, 2, 0.9572 ** 2), (1, 2, 1.5139 ** 2))
        im = 1.0 / m[w0:].reshape(-1, 3)
        frc = _plain_pairs(s, x, q)[0]
        for _ in range(case["steps"]):
            v = v * lam + frc / m * dt
            new = x + v * dt
            if s.n_waters:
                old, p = x[w0:].reshape(-1, 3, 3), new[w0:].reshape(-1, 3, 3).clone()
                for _it in range(60):
                    for a, b, d2 in cons:
                        dp, do = p[:, a] - p[:, b], old[:, a] - old[:, b]
                        g = (d2 - (dp * dp).sum(-1)) / (2 * (im[:, a] + im[:, b]) * (dp * do).sum(-1))
                        p[:, a] += (g * im[:, a])[:, None] * do
                        p[:, b] -= (g * im[:, b])[:, None] * do
                new = torch.cat((new[:w0], p.reshape(-1, 3)))
                v = torch.cat((v[:w0], (new[w0:] - x[w0:]) / dt))
            x = new
            kT = float((m * v * v).sum()) / ndof
            lam = math.sqrt(min(max(1.0 + 0.2 * (kT0 / kT - 1.0), 0.64), 1.5625))
            frc, e_lj, e_c, vir = _plain_pairs(s, x, q)
        hist = np.bincount(s.atom_type, minlength=s.n_types).astype(np.float64)
        k = S.lj_type_index(np.arange(s.n_types)[:, None], np.arange(s.n_types)[None, :])
        c6 = float((hist[:, None] * hist[None, :] * s.pair_B.astype(np.float64)[k]).sum())
        long_range = -2.0 / 3.0 * math.pi * c6 / s.cutoff ** 3 / 6.0 / s.volume
        all_energies.append([float(e_lj.sum()), long_range, float(e_c.sum())] + vir.sum(0).tolist())
        states.append((x.cpu().numpy(), v.cpu().numpy(), frc.cpu().numpy()))
    return _joined(np.array(all_energies), states)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    fep = _fep(case, seed) if kind == "soft" else None
    s = fep.system() if fep is not None else _system(case, seed)
    x = torch.from_numpy(s.crd.astype(np.float32)).cuda().double()
    q = torch.from_numpy(s.charge.astype(np.float32)).cuda().double()
    frc, e_lj, e_c, vir = _soft_pairs(fep, s, x, q) if fep is not None else _plain_pairs(s, x, q)
    out = {}
    terms = case.get("terms", "f")
    if terms != "f":
        out["totals"] = torch.cat((torch.stack((e_lj.sum(), e_c.sum())), vir.sum(0)))
    if terms == "fev":
        # a water's sites hand theirs to its first atom
        first = _molecules(s)
        first = torch.searchsorted(first, first)
        give = lambda a: torch.zeros_like(a).index_add_(0, first, a)  # noqa: E731
        e_lj, e_c, vir = give(e_lj), give(e_c), give(vir)
        out["direct"] = e_c
    energy = e_lj + e_c
    if case.get("fused"):
        _excluded(s, x, q, frc, energy, vir)
    out["frc"] = frc
    if terms == "fev":
        out["energy"] = energy
        out["virial"] = vir
    if case.get("full_list"):
        out.update(counts=None, lists=None, overflow=None)
    return out
