"""The energy sums of non-water atoms on the mixed path hold every pair's energy to far below FP32's
rounding of the largest: a charge whose neighbours come in mirror-image pairs of opposite charge, 1,712
kcal/mol each, which cancel bit by bit, and 200 weak neighbours of about 0.1 kcal/mol.  What is left
is the weak pairs' energy, each within a few FP32 roundings of itself; sums that hold a strong and a
weak pair in one FP32 number are off by up to half a unit in the last place of 1,712, 6e-5, at every
addition."""
import numpy as np
import pytest

from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, Nonbonded

pytestmark = pytest.mark.gpu


def test_weak_pairs_beside_cancelling_strong_ones():
    rng = np.random.Generator(np.random.PCG64(3))
    box = 40.0
    u = rng.normal(size=(20, 3))
    strong = np.round(2.0 * u / np.linalg.norm(u, axis=1)[:, None] * 1024) / 1024      # exact in FP32
    v = rng.normal(size=(200, 3))
    weak = rng.uniform(4.0, 7.0, (200, 1)) * v / np.linalg.norm(v, axis=1)[:, None]
    q = np.concatenate([[2000.0, -2000.0], np.full(20, 0.016), np.full(20, -0.016), np.full(100, 1e-4), np.full(100, -3e-5)])
    q[1] -= q.sum()
    xyz = np.concatenate([[[0.0, 0.0, 0.0], [20.0, 20.0, 20.0]], strong, -strong, weak])
    b = S._Builder(arith=True)
    for x, c in zip(xyz, q):
        b.add_monomer(x[None, :], [c], [0.0], [0.0], S.MON_OTHER)
    s = b.finish("mirror", box, rvmx=9.0, relx=9.0, alpha=0.35, nfft=(40, 40, 40), seed=3)
    direct = []
    for precision in (MOIL_NB_MIXED, MOIL_NB_FP64):
        nb = Nonbonded(s, precision=precision)
        e = nb.eforce(s.coor)[1]
        direct.append(e["e_el"] + e["e_lsym"])
        nb.close()
    # 8 FP32 roundings of every other pair: magnitudes of 22.5 (the weak ones) and 10.7 kcal/mol (the rest)
    assert abs(direct[0] - direct[1]) <= 8 * 2.0 ** -24 * 33.2
