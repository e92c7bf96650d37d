"""The rules that split a cluster's work over warps, at the sizes where they
change: the force kernel's parts of a list, the search's and the pruning's
teams of four warps (and a team's staging when it overflows), and the bound
on cluster pairs that one periodic image serves.  Lists against the oracle
pair for pair; forces against the FP64 sum over that list.
"""
import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu

# FP32 pair arithmetic: 1e-6 relative RMS against FP64 on every system of the
# parity tests, which hold it to the same bound
FORCE_REL_RMS_TOL = 1e-5


def _water(n_waters, cutoff, seed, box=None, **kw):
    from spgnb import systems as S
    L = box or ((n_waters + kw.get("n_solute", 0)) / 0.0334) ** (1.0 / 3.0)
    return S.water_system(n_waters, L, seed, cutoff=cutoff, skin=2.0, **kw)


CASES = {
    # the force kernel's 16, 8, 4, 2 and 1 parts (fewer in the energy modes)
    "parts-16": lambda: _water(520, 8.0, 41),
    "parts-8": lambda: _water(900, 8.0, 42),
    "parts-4": lambda: _water(1700, 8.0, 43, n_solute=50),
    "parts-2": lambda: _water(3100, 8.0, 44),
    # one warp and four warps a cluster, either side of the line
    "team-4": lambda: _water(3650, 8.0, 45),
    "team-1": lambda: _water(4600, 8.0, 46),
    "parts-1": lambda: _water(5600, 8.0, 52),
    # a skewed cell large enough for a warp a cluster
    "triclinic-team-1": lambda: _water(5200, 8.0, 47, box=(53.0, 56.5, 59.0), n_solute=150,
                                       angles=(75.0, 80.0, 70.0)),
    # twice water's density at the longest cutoff: a warp's share of a
    # cluster's candidates and words exceeds what it can stage
    "dense": lambda: _water(1800, 12.0, 48, box=30.0),
    # boxes at and below twice the list radius: cluster pairs need their own images
    "box-2-radii": lambda: _water(290, 8.0, 49, box=20.2),
    "box-1.6-radii": lambda: _water(140, 8.0, 50, box=16.1),
    "box-oblong": lambda: _water(400, 8.0, 51, box=(21.0, 23.0, 25.0)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_split_lists_and_forces(torch_cuda, oracle, name):
    from spgnb.engine import PlainPath
    s = CASES[name]()
    p = PlainPath(s, export_atom_groups=True, max_neighbor_numbers=3000)
    for _ in range(8):  # the dense box starts above the default capacities
        if not p.nl.Check_Overflow({}, 149, s.cell, s.rcell):
            break
        p.update(0, forced=True)
        p.force()
    assert p.nl.stats()["overflow"] == 0
    counts, lists = p.nl.host_atom_groups()
    oc, ol = oracle.nl_build(s, mode=1)
    assert np.array_equal(counts, oc)
    assert np.array_equal(lists, ol)
    ref = oracle.pair_force(s, oc, ol, per_atom=False)
    for energy, per_atom in ((False, False), (True, False), (True, True)):
        frc = p.force(need_energy=energy, need_virial=energy, per_atom=per_atom).cpu().numpy()
        assert rel_rms(frc, ref["frc"]) <= FORCE_REL_RMS_TOL
        if not energy:
            continue
        tot = p.lj.totals()
        scale = abs(ref["e_lj"]) + abs(ref["e_coul"])
        assert abs(tot[0] - ref["e_lj"]) <= 1e-5 * scale
        assert abs(tot[1] - ref["e_coul"]) <= 1e-5 * scale
        assert np.abs(tot[2:] - ref["virial"]).max() <= 1e-5 * np.abs(ref["virial"]).max()
        if per_atom:
            # the per-atom arrays hold the same pairs: N FP32 values summed
            assert abs(p.atom_energy.double().sum().item() - tot[0] - tot[1]) <= 1e-6 * scale
            assert np.abs(p.atom_virial.double().sum(0).cpu().numpy() - tot[2:]).max() <= 1e-6 * np.abs(tot[2:]).max()


@pytest.mark.parametrize("beta", [0.0, 0.002, 0.01, 0.2, 0.34, 0.5])
def test_ewald_fit_routes(torch_cuda, oracle, beta):
    """The pair function's fits over the Ewald parameters that take each form:
    in w (none, tiny), scaled to the system, and erfc past the fits' range."""
    from dataclasses import replace
    from spgnb.engine import PlainPath
    s = replace(_water(700, 8.0, 53, n_solute=40), beta=beta)
    p = PlainPath(s, export_atom_groups=True)
    counts, lists = p.nl.host_atom_groups()
    ref = oracle.pair_force(s, counts, lists, per_atom=False)
    for energy in (False, True):
        frc = p.force(need_energy=energy, need_virial=energy, per_atom=False).cpu().numpy()
        assert rel_rms(frc, ref["frc"]) <= FORCE_REL_RMS_TOL
    tot = p.lj.totals()
    assert abs(tot[1] - ref["e_coul"]) <= 1e-5 * (abs(ref["e_lj"]) + abs(ref["e_coul"]))
