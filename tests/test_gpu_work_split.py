"""The rules that split a cluster's work over warps, at the sizes where they
change: the force kernel's parts of a list, the search's teams of four and two
warps and the pruning's of four (and a team's staging when it overflows), and
the bound on cluster pairs that one periodic image serves.  Lists against the
oracle pair for pair; forces against the FP64 sum over that list.  Every case
also states the split it is there for, read from the launched kernels, so that
a rule that moves fails here instead of leaving a form untested.
"""
import numpy as np
import pytest

from conftest import in_fresh_process, kernel_launches, rel_rms

pytestmark = pytest.mark.gpu

# FP32 pair arithmetic: 1e-6 relative RMS against FP64 on every system of the
# parity tests, which hold it to the same bound
FORCE_REL_RMS_TOL = 1e-5


def _water(n_waters, cutoff, seed, box=None, **kw):
    from spgnb import systems as S
    L = box or ((n_waters + kw.get("n_solute", 0)) / 0.0334) ** (1.0 / 3.0)
    return S.water_system(n_waters, L, seed, cutoff=cutoff, skin=2.0, **kw)


# each: the system, then on a chip of 148 SMs the parts of a list in the force
# kernel (fewer in the energy modes) and the warps a cluster in the search and
# in the pruning.  Clusters an SM at the lines: 16 and 32 (search), 36 (pruning).
CASES = {
    "parts-16": (lambda: _water(520, 8.0, 41), 16, 4, 4),
    "parts-8": (lambda: _water(900, 8.0, 42), 8, 4, 4),
    "parts-4": (lambda: _water(1700, 8.0, 43, n_solute=50), 4, 4, 4),
    "parts-2": (lambda: _water(3100, 8.0, 44), 2, 4, 4),
    # below and above sixteen clusters an SM
    "search-4": (lambda: _water(3650, 8.0, 45), 2, 4, 4),
    "search-2": (lambda: _water(4600, 8.0, 46), 2, 2, 4),
    "parts-1": (lambda: _water(5600, 8.0, 52), 1, 2, 4),
    # above 32, and above 36
    "search-1": (lambda: _water(8400, 8.0, 54), 1, 1, 4),
    "prune-1": (lambda: _water(9300, 8.0, 55), 1, 1, 1),
    # skewed cells, with a team and with a warp a cluster
    "triclinic-2": (lambda: _water(5200, 8.0, 47, box=(53.0, 56.5, 59.0), n_solute=150, angles=(75.0, 80.0, 70.0)),
                    2, 2, 4),
    "triclinic-1": (lambda: _water(10000, 8.0, 56, box=(66.0, 70.3, 73.4), n_solute=150, angles=(75.0, 80.0, 70.0)),
                    1, 1, 1),
    # twice water's density at the longest cutoff: a warp's share of a
    # cluster's candidates and words exceeds what it can stage; and two warps'
    # shares at water's density
    "dense": (lambda: _water(1800, 12.0, 48, box=30.0), 8, 4, 4),
    "search-2-staging": (lambda: _water(7000, 12.0, 57), 1, 2, 4),
    # boxes at and below twice the list radius: cluster pairs need their own images
    "box-2-radii": (lambda: _water(290, 8.0, 49, box=20.2), 16, 4, 4),
    "box-1.6-radii": (lambda: _water(140, 8.0, 50, box=16.1), 16, 4, 4),
    "box-oblong": (lambda: _water(400, 8.0, 51, box=(21.0, 23.0, 25.0)), 16, 4, 4),
}


def _split(launches):
    """(parts of a list, warps a cluster in the search, in the pruning) of a
    build and its first force-only call."""
    one = {}
    for kernel in ("k_search", "k_prune8", "k_pair8"):
        found = [k for k in launches if kernel in k["name"]]
        assert len(found) == 1, (kernel, [k["name"] for k in launches])
        one[kernel] = found[0]
    clusters = one["k_search"]["grid"][0]  # a block a cluster (below the bound on one-warp blocks)
    parts, rest = divmod(one["k_pair8"]["grid"][0], clusters)
    assert rest == 0
    return parts, one["k_search"]["block"][0] // 32, int(one["k_prune8"]["name"].split("k_prune8<")[1][0])


def _path(s, **kw):
    from spgnb.engine import PlainPath
    p = PlainPath(s, **kw)
    for _ in range(8):  # the dense box starts above the default capacities
        if not p.nl.Check_Overflow({}, 149, s.cell, s.rcell):
            break
        p.update(0, forced=True)
        p.force()
    assert p.nl.stats()["overflow"] == 0
    return p


def traced_splits():
    """Every case's split, read from its launched kernels."""
    import torch
    out = {}
    for name, (make, *_) in CASES.items():
        p = _path(make())

        def build_and_force():
            p.update(0, forced=True)
            p.force()

        out[name] = _split(kernel_launches(torch, build_and_force))
    return out


def test_cases_run_the_splits_they_are_for(torch_cuda):
    assert torch_cuda.cuda.get_device_properties(0).multi_processor_count == 148, "the cases' sizes are for 148 SMs"
    got = in_fresh_process("test_gpu_work_split", "traced_splits")
    assert {k: tuple(v) for k, v in got.items()} == {k: tuple(split) for k, (_, *split) in CASES.items()}


@pytest.mark.parametrize("name", list(CASES))
def test_split_lists_and_forces(torch_cuda, oracle, name):
    s = CASES[name][0]()
    p = _path(s, export_atom_groups=True, max_neighbor_numbers=3000)
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


def test_two_sided_team_staging(torch_cuda):
    """A two-sided table past what a team of four can stage holds the pairs of
    the one-sided one: the full lists that the two give are the same."""
    from spgnb.engine import SoftCorePath
    from spgnb import systems as S
    p = SoftCorePath(S.fep_system(_water(1750, 16.0, 58, box=36.2, n_solute=60), n_perturbed=8))
    full = []
    for dhdl in (False, True):
        for _ in range(8):  # the box starts above the default capacities
            p.force()
            if dhdl:
                p.dhdl()
            if not p.nl.Check_Overflow({}, 149, p.cell, p.rcell):
                break
            p.update(0, forced=True)
        counts, lists, overflow = p.nl.build_full(p.n, p.crd, p.cell, p.rcell, 0.0, 4000)
        stats = p.nl.stats()
        assert stats["overflow"] == 0 and int(overflow.item()) == 0
        # four shares of 128 elements: past this on average, some cluster's overflow
        assert not dhdl or stats["entries"] > 4 * 128 * stats["clusters"]
        counts, lists = counts.cpu().numpy(), lists.cpu().numpy()
        full.append([np.sort(lists[i, :counts[i]]) for i in range(p.n)])
    assert all(np.array_equal(a, b) for a, b in zip(*full))


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
