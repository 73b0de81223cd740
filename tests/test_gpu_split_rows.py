"""Pair kernels that share one water's or atom's list among the lanes of a warp, at the sizes
where the sharing can go wrong: water counts that do not fill the last block, rows shorter and
longer than a warp's buffer, solutes of a few atoms.  Each against the oracle in parity mode:
the FP64 path to 2^-25 of the gradient (its 2 alpha / sqrt(pi) is an FP32 constant) and 1e-10 of
the energy-term scale per term."""
import numpy as np
import pytest

from conftest import ENERGY_TERMS, energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def dense_cluster(n, seed, shrink):
    """n waters at liquid density with every oxygen moved toward the centre of the box, so the
    rows of the middle grow past a full shell."""
    s = S.water_box(n, (n / S.WATER_DENSITY) ** (1 / 3), seed, name="cluster")
    xyz = s.coor.reshape(-1, 3, 3)
    s.coor = (xyz - shrink * xyz[:, 0, :][:, None, :]).reshape(-1, 3)
    return s


SYSTEMS = {
    "lone_water": lambda: S.water_box(1, 20.0, 3),
    "three_waters": lambda: S.water_box(3, 18.7, 4),
    "197_waters": lambda: S.water_box(197, 18.1, 5),
    "1003_waters": lambda: S.water_box(1003, (1003 / S.WATER_DENSITY) ** (1 / 3), 6),
    "dense_rows": lambda: dense_cluster(900, 7, 0.25),
    "solute": lambda: S.config1(seed=7, n_solute=61, n_ions=7, n_waters=299, box=24.0),
    "solute_geometric": lambda: S.config1(seed=8, n_solute=45, n_ions=7, n_waters=150, box=24.0, arith=False,
                                          tiny_h=True),
}


@pytest.mark.parametrize("name", SYSTEMS)
def test_split_rows_match_oracle(name, precision=MOIL_NB_FP64):
    s = SYSTEMS[name]()
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, precision=precision)
    for _ in range(2):                      # the build, then list reuse
        dpot, e = nb.eforce(s.coor)
        if eref["site_pairs"] == 0:
            # no pairs: gradient and total are small remainders of cancelling terms
            assert np.abs(dpot - ref).max() <= 1e-6 * energy_scale(eref)
            assert abs(e["e_total"] - eref["e_total"]) <= 1e-6 * energy_scale(eref)
        else:
            assert rel_rms(dpot, ref) <= 2.0 ** -25
            assert all(abs(e[k] - eref[k]) <= 1e-10 * energy_scale(eref) for k in ENERGY_TERMS)
    assert nb.pair_stats()["site_pairs"] == eref["site_pairs"]
    nb.close()
