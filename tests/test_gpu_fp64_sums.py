"""The FP64 path's fixed-point gradient holds what one rounding to 2^-33 kcal/mol/Å leaves, whatever the number
of pairs: LJ alone (no charges, so no spline grid and no FP32 constant takes part) against the oracle.
Bound: half of that unit again for the finer rounding of the waters' parts (2^-43 each, some hundreds
at most) and FP64 arithmetic."""
import numpy as np
import pytest

from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def uncharged(s):
    s = s.copy()
    s.ptchg[:] = 0.0
    s.p14[:, 2] = 0.0
    return s


@pytest.mark.parametrize("name", ["waters_216", "waters_1334", "solute"])
def test_gradient_is_rounded_once(name):
    s = uncharged({"waters_216": lambda: S.config0(), "waters_1334": lambda: S.water_box(1334, 34.2, 4),
                   "solute": lambda: S.config1(seed=7, n_solute=61, n_ions=7, n_waters=299, box=24.0)}[name]())
    ref = O.eforce(s, mode="parity")[0]
    nb = Nonbonded(s, precision=MOIL_NB_FP64)
    for _ in range(2):
        dpot = nb.eforce(s.coor)[0]
        assert np.abs(dpot - ref).max() <= 1.5 * 2.0 ** -33 + 1e-14 * np.abs(ref).max()
    nb.close()


def test_large_forces_take_the_coarse_array():
    """Two oxygens 0.9 Å apart: a force of 10^8 kcal/mol/Å, beyond the fine array's parts, beside ordinary ones."""
    s = uncharged(S.config0())
    x = s.coor.reshape(-1, 3, 3)
    x[5] += x[9, 0] + [0.9, 0.0, 0.0] - x[5, 0]
    s.coor = x.reshape(-1, 3)
    ref = O.eforce(s, mode="parity")[0]
    assert np.abs(ref).max() > 1e7
    nb = Nonbonded(s, precision=MOIL_NB_FP64)
    dpot = nb.eforce(s.coor)[0]
    nb.close()
    # FP64 rounding of the largest force's own terms, relative to each atom's force
    assert (np.abs(dpot - ref) <= 1.5 * 2.0 ** -33 + 1e-12 * np.abs(ref).max(1, keepdims=True)).all()
