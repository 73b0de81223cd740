"""Pair kernels that share one water's or atom's list among the lanes of a warp, at the sizes
where the sharing can go wrong: water counts that do not fill the last block, rows shorter and
longer than a warp's buffer, solutes of a few atoms.  Each against the oracle in parity mode:
the FP64 path to 2^-25 of the gradient (its 2 alpha / sqrt(pi) is an FP32 constant) and 1e-10 of
the energy-term scale per term, the mixed path to 1e-5 of the gradient and 1e-6 of that scale."""
import numpy as np
import pytest

from conftest import ENERGY_TERMS, energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, WATER_FULL, WATER_HALF, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def dense_cluster(n, seed, shrink):
    """n waters at liquid density with every oxygen moved toward the centre of the box, so the
    rows of the middle grow past a full shell."""
    s = S.water_box(n, (n / S.WATER_DENSITY) ** (1 / 3), seed, name="cluster")
    xyz = s.coor.reshape(-1, 3, 3)
    s.coor = (xyz - shrink * xyz[:, 0, :][:, None, :]).reshape(-1, 3)
    return s


def hydrogens_with_lj(s):
    """The same system with LJ coefficients on the waters' hydrogens, which meet non-water atoms."""
    h = np.arange(s.npt - 3 * 150, s.npt).reshape(-1, 3)[:, 1:].ravel()
    s.epsgm12, s.epsgm6 = s.epsgm12.copy(), s.epsgm6.copy()
    s.epsgm12[h], s.epsgm6[h] = 0.4, 0.6
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
    "solute_hydrogen_lj": lambda: hydrogens_with_lj(S.config1(seed=9, n_solute=45, n_ions=7, n_waters=150, box=24.0)),
}


def close_to_oracle(dpot, e, ref, eref, precision):
    scale = energy_scale(eref)
    fp64 = precision == MOIL_NB_FP64
    assert all(abs(e[k] - eref[k]) <= (1e-10 if fp64 else 1e-6) * scale for k in ENERGY_TERMS + ("e_total",))
    if eref["site_pairs"] == 0:
        # no pairs: the gradient is a small remainder of cancelling terms
        assert np.abs(dpot - ref).max() <= 1e-6 * scale
    else:
        assert rel_rms(dpot, ref) <= (2.0 ** -25 if fp64 else 1e-5)


@pytest.mark.parametrize("precision", [MOIL_NB_FP64, MOIL_NB_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", SYSTEMS)
def test_split_rows_match_oracle(name, precision):
    s = SYSTEMS[name]()
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, precision=precision)
    for _ in range(2):                      # the build, then list reuse
        dpot, e = nb.eforce(s.coor)
        close_to_oracle(dpot, e, ref, eref, precision)
    assert nb.pair_stats()["site_pairs"] == eref["site_pairs"]
    nb.close()


@pytest.mark.parametrize("filler", [1, 11], ids=["8_lanes", "4_lanes"])
def test_long_rows_on_full_lists(filler):
    """Rows of more than 64 entries per lane, in handles of more than 4,096 and 32,768 waters (8
    and 4 lanes per water), beside a replica that ends inside a block."""
    dense = dense_cluster(1001, 9, 0.5)
    box = S.water_box(3203, (3203 / S.WATER_DENSITY) ** (1 / 3), 10)
    nb = Nonbonded([dense] + [box] * filler, shape=dict(water_kernel=WATER_FULL), groups=1)
    dps, es = nb.eforce()
    for k, s in ((0, dense), (filler, box)):
        ref, eref = O.eforce(s, mode="parity")
        close_to_oracle(dps[k], es[k], ref, eref, MOIL_NB_MIXED)
    nb.close()


@pytest.mark.parametrize("n", [1215, 1217, 1275])
def test_more_partners_than_shared_accumulators(n):
    """Half lists keep 9.5 partner accumulators per water of a block in shared memory: with blocks
    of 128 waters 1,216, and the shares of the partners beyond go straight to the gradient."""
    s = dense_cluster(n, 11, 0.55)
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, shape=dict(water_kernel=WATER_HALF, half_block=128))
    for _ in range(2):
        dpot, e = nb.eforce(s.coor)
        close_to_oracle(dpot, e, ref, eref, MOIL_NB_MIXED)
    assert nb.shape()["water_kernel"] == WATER_HALF
    nb.close()


@pytest.mark.parametrize("precision", [MOIL_NB_FP64, MOIL_NB_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["lone_water", "197_waters", "dense_rows", "solute"])
def test_pressure_rows_match_oracle(name, precision):
    """Pressure terms where a water's owned pairs end inside eight lanes and where they fill its
    buffer of 64 more than once: 1e-5 (mixed) and 1e-9 (FP64) of the tensor's magnitude sum."""
    s = SYSTEMS[name]()
    mol, mass = S.molecules(s)
    want = O.pressure(s, mol, mass, mode="mi")[2]
    nb = Nonbonded(s, precision=precision)
    nb.set_molecules(mol, mass)
    press = nb.pressure(s.coor)[2]
    nb.close()
    assert np.abs(press - want).max() <= (1e-9 if precision == MOIL_NB_FP64 else 1e-5) * np.abs(want).sum()


def test_pass_is_redone_with_its_evaluation():
    """Derivatives and pressure as a handle's first call, on rows that overflow their first capacity
    (the evaluation and the pass queued behind it are redone), and again on the lists then built."""
    s = dense_cluster(900, 12, 0.55)
    mol, mass = S.molecules(s)
    for call in (lambda nb: np.stack(nb.adjoint(s.coor)), lambda nb: nb.pressure(s.coor)[2]):
        nb = Nonbonded(s)
        nb.set_molecules(mol, mass)
        first, again = call(nb), call(nb)
        nb.close()
        assert np.isfinite(first).all() and np.abs(first - again).max() <= 1e-9 * np.abs(again).max()
