"""Derivative and pressure passes are queued behind an evaluation before its status is known.  Where the lists
turn out stale (sites moved past half the skin since the build) both are redone: the results are those of
a handle whose first call has these coordinates, to the FP32 paths' rounding.  And half lists whose
blocks have more partners than their shared accumulators, for the block sizes of 256 and 512 waters."""
import numpy as np
import pytest

from conftest import ENERGY_TERMS, energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, WATER_HALF, Nonbonded
from oracle import oracle as O
from test_gpu_split_rows import dense_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("name", ["waters", "solute"])
def test_pass_behind_a_stale_evaluation(name, precision):
    s = S.config0() if name == "waters" else S.config1(seed=7, n_solute=61, n_ions=7, n_waters=299, box=24.0)
    mol, mass = S.molecules(s)
    rng = np.random.Generator(np.random.PCG64(8))
    moved = s.coor.copy()
    w = s.npt - 3 * s.nwaters
    moved[w:] += np.repeat(rng.uniform(-0.6, 0.6, (s.nwaters, 3)), 3, axis=0)      # far past half the skin
    for call in (lambda nb, x: np.concatenate(nb.adjoint(x)), lambda nb, x: np.concatenate([nb.pressure(x)[2]]),
                 lambda nb, x: nb.pressure(x)[0]):
        fresh, used = Nonbonded(s, precision=precision, skin=0.2), Nonbonded(s, precision=precision, skin=0.2)
        for nb in (fresh, used):
            nb.set_molecules(mol, mass)
        want = call(fresh, moved)
        call(used, s.coor)
        call(used, s.coor)              # replayed without a rebuild
        got = call(used, moved)         # replayed without a rebuild, dropped and redone
        fresh.close()
        used.close()
        assert np.isfinite(got).all() and rel_rms(got, want) <= (1e-11 if precision == MOIL_NB_FP64 else 2e-6)


@pytest.mark.parametrize("hb,n,shrink", [(256, 2432, 0.55), (256, 2600, 0.55), (256, 4870, 0.55), (512, 3700, 0.55),
                                         (512, 6200, 0.5)])
def test_partners_beyond_the_shared_accumulators(hb, n, shrink):
    """Up to 2,432 partners of a block have accumulators with 256 waters per block, 4,864 with 512; the blocks
    here have 2,429, 2,579, 3,274, 3,274 and 5,067."""
    s = dense_cluster(n, 13, shrink)
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, shape=dict(water_kernel=WATER_HALF, half_block=hb))
    for _ in range(2):
        dpot, e = nb.eforce(s.coor)
        assert rel_rms(dpot, ref) <= 1e-5
        assert all(abs(e[k] - eref[k]) <= 1e-6 * energy_scale(eref) for k in ENERGY_TERMS + ("e_total",))
    assert nb.shape()["water_kernel"] == WATER_HALF
    nb.close()
