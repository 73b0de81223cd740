"""More replicas in one handle than a grid's second axis holds (65,535): evaluation, derivatives and
pressure of 65,600 copies of a box of two waters.  Each against the oracle: gradient and derivatives 1e-5,
energies 1e-6 of the term scale, pressure 1e-5 of the tensor's magnitude sum."""
import numpy as np
import pytest

from conftest import energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu

REPLICAS = 65600


def test_more_replicas_than_a_grid_axis():
    s = S.water_box(2, 9.0, 3, rc=4.0, nfft=(8, 8, 8))
    s.coor[3:] += s.coor[0] - s.coor[3] + [2.4, 1.6, 0.9]          # 3.0 Å apart
    mol, mass = S.molecules(s)
    nb = Nonbonded([s] * REPLICAS, skin=0.3)
    nb.set_molecules(np.tile(mol, REPLICAS), np.tile(mass, REPLICAS))
    ref, eref = O.eforce(s, mode="parity")
    dps, es, press = nb.pressure()
    assert rel_rms(np.stack(dps), np.broadcast_to(ref, (REPLICAS,) + ref.shape)) <= 1e-5
    assert max(abs(e["e_total"] - eref["e_total"]) for e in es) <= 1e-6 * energy_scale(eref)
    want = O.pressure(s, mol, mass, mode="mi")[2]
    assert np.abs(np.stack(press) - want).max() <= 1e-5 * np.abs(want).sum()
    for got, w in zip(nb.adjoint(), O.adjoint(s)):
        assert rel_rms(np.stack(got), np.broadcast_to(w, (REPLICAS, len(w)))) <= 1e-5
    nb.close()
