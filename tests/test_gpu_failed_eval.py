"""An evaluation through host buffers that fails leaves the caller's gradient as it was (handles without
replica groups), and the handle works on."""
import numpy as np
import pytest

from conftest import rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, MoilNbError, Nonbonded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [True, False], ids=["first_call", "later_call"])
@pytest.mark.parametrize("fault", ["nan", "hydrogen_far"])
@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
def test_gradient_untouched_by_a_failed_evaluation(precision, fault, first):
    s = S.config0()
    nb = Nonbonded(s, precision=precision)
    good = nb.eforce(s.coor)[0] if not first else None
    bad = s.coor.copy()
    if fault == "nan":
        bad[300, 1] = np.nan
    else:
        bad[301] = bad[300] + [1.2, 0.0, 0.0]
    dpot = np.random.Generator(np.random.PCG64(1)).normal(size=s.coor.shape)
    before = dpot.copy()
    with pytest.raises(MoilNbError):
        nb.eforce_into(bad, dpot)
    assert np.array_equal(dpot, before)
    again = nb.eforce(s.coor)[0]
    assert np.isfinite(again).all() and (good is None or rel_rms(again, good) <= 1e-6)
    nb.close()
