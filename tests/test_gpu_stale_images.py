"""Pairs near half a box on a list older than their motion: the build-time
list's pairs are evaluated at their minimum image at the current coordinates,
as the reference does, also where that is another image than at the build."""
from dataclasses import replace

import numpy as np
import pytest


# box length, distance of a pair at the build, how far its second atom then
# moves away, and the distance along the axis of an atom without interactions
# beside each (0: none, every cluster a point).  List radius 10, cutoff 8: each
# pair is listed, and ends inside the cutoff by its other image.
CASES = {"points-2-radii": (20.0, 9.9, 2.15, 0.0), "clusters-2.1-radii": (21.0, 9.95, 3.5, 0.4)}


def _pairs_along_the_axes(L, gap, drift, width):
    """A pair of atoms along each axis of a cube, every one alone in its grid
    cell but for its companion; the system, the pairs and the coordinates
    after the drift."""
    from spgnb import systems as S
    first = np.array([[0.05, 2.5, 2.5], [7.5, 10.05, 12.5], [17.5, 7.5, 0.05]])
    crd, moved, kind, pairs = [], [], [], []
    for axis, x in enumerate(first):
        u = np.eye(3)[axis]
        pairs.append((len(crd), len(crd) + 1))
        crd += [x, x + gap * u]
        moved += [x, x + (gap + drift) * u]
        kind += [0, 0]
        if width:
            crd += [x + width * u, x + (gap + width) * u]
            moved += crd[-2:]
            kind += [1, 1]
    n = len(crd)
    A, B = S.lj_pair_tables([3.2, 3.2], [0.3, 0.0])
    none, one = np.zeros(n, np.int32), np.ones(n, np.int32)
    t = S.water_system(1, L, 1, cutoff=8.0, skin=2.0)
    s = replace(t, crd=np.array(crd, np.float32), vel=np.zeros((n, 3), np.float32), charge=np.zeros(n, np.float32),
                atom_type=np.array(kind, np.int32), pair_A=A, pair_B=B, n_types=2, excl_start=none, excl_numbers=none,
                excl_list=np.zeros(0, np.int32), mass=12 * np.ones(n, np.float32),
                res_start=np.arange(n, dtype=np.int32), res_len=one, n_solute=n)
    return s, pairs, np.array(moved, np.float32)


@pytest.mark.parametrize("name", list(CASES))
def test_the_moved_pairs_meet_through_their_other_image(oracle, name):
    """The inputs do what they are for (the oracle alone)."""
    L, gap, drift, width = CASES[name]
    s, pairs, moved = _pairs_along_the_axes(L, gap, drift, width)
    counts, lists = oracle.nl_build(s, mode=1)
    for i, j in pairs:
        k0 = int(np.sum(counts[:i]))
        assert j in lists[k0:k0 + counts[i]]
        d = (moved[j] - moved[i]).astype(np.float64)
        assert np.linalg.norm(d) > s.cutoff > np.linalg.norm(d - L * np.round(d / L))


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_pairs_take_their_image_at_the_current_coordinates(torch_cuda, oracle, name):
    from spgnb.engine import PlainPath
    s, pairs, moved = _pairs_along_the_axes(*CASES[name])
    p = PlainPath(s, refresh_interval=1000, solvent=False)
    mc = torch_cuda.from_numpy(moved).cuda()
    p.update(1, crd=mc)  # not a rebuild step
    counts, lists = oracle.nl_build(s, mode=1)
    ref = oracle.pair_force(s, counts, lists, crd=moved)
    assert all(np.linalg.norm(ref["frc"][i]) > 0 for pair in pairs for i in pair)
    for energy in (False, True):
        frc = p.force(need_energy=energy, need_virial=energy, crd=mc).cpu().numpy()
        # FP32 pairs: 1e-6 of a term, a few terms an atom
        assert np.abs(frc - ref["frc"]).max() <= 1e-5 * np.abs(ref["frc"]).max()
