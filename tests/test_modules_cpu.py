"""Argument checks of the Python module mirrors that need no device."""
import numpy as np
import pytest


def _solvent_call(**bad):
    """The solvent module's force call over an spgnb list, one argument replaced."""
    from spgnb.modules import NEIGHBOR_LIST, SOLVENT_LENNARD_JONES
    solvent = SOLVENT_LENNARD_JONES()
    solvent.is_initialized, solvent.handle = True, 1
    nl = NEIGHBOR_LIST()
    nl.handle = 1  # a list made by the library: the LJ module's call does the work
    cell = np.array([20, 0, 20, 0, 0, 20], np.float32)
    args = dict(atom_numbers=6, residue_numbers=2, d_res_start=None, crd=None, charge=None, frc=None, cell=cell,
                rcell=1 / np.maximum(cell, 1), nl=nl, pme_beta=0.3, need_atom_energy=False, atom_energy=None,
                need_virial=False, atom_lj_virial=None, atom_direct_pme_energy=None)
    try:
        return solvent.LJ_PME_Direct_Force_With_Atom_Energy_And_Virial(**{**args, **bad})
    finally:
        solvent.handle = nl.handle = None


def test_solvent_call_over_an_spgnb_list_does_nothing():
    assert _solvent_call() is None


@pytest.mark.parametrize("name", ["atom_numbers", "residue_numbers", "cell", "rcell", "pme_beta", "need_atom_energy",
                                  "need_virial"])
def test_solvent_call_over_an_spgnb_list_refuses_wrong_types(name):
    with pytest.raises((TypeError, ValueError)):
        _solvent_call(**{name: "six"})
