"""Replicas of 65,536 waters or more, whose water rows hold 32-bit entries: every kernel over those rows
(both precisions' water kernels, derivatives, pressure).  The box is a small one repeated three times along
each axis with three times the grid, so its gradient and derivatives are the small box's 27 times over and
its energies and pressure terms 27 times as large: the oracle works on the small box.  Tolerances of
the 16-bit rows: gradient 1e-5 (mixed), 2^-25 (FP64, whose 2 alpha / sqrt(pi) is an FP32 constant); energies
1e-6 / 1e-10 of the term scale, derivatives 1e-5 of their norm, pressure 1e-5 of the tensor's magnitude sum."""
import dataclasses

import numpy as np
import pytest

from conftest import energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu

M = 3


def small_box(seed=31):
    """2,470 waters and two ions of opposite charge in 42 Å, on a 36^3 grid."""
    rng = np.random.Generator(np.random.PCG64(seed))
    L = 42.0
    sites = S._lattice_sites(14, L)
    pick = np.sort(rng.choice(len(sites), size=2472, replace=False))
    oxy = sites[pick] + rng.uniform(-0.3, 0.3, (2472, 3))
    b = S._Builder(arith=True)
    for x, q in zip(oxy[[100, 2100]], (1.0, -1.0)):
        b.add_monomer(x[None, :], [q], [0.0469], [S.rmin2_to_sigma(1.3638)], S.MON_ION)
    b.add_waters(S._place_waters(rng, np.delete(oxy, [100, 2100], axis=0)))
    return b.finish("small", L, rvmx=9.0, relx=9.0, alpha=0.35, nfft=(36, 36, 36), seed=seed)


def repeated(s):
    n, L = s.npt, np.array(s.box)
    shifts = [(np.array([i, j, k]) - 1) * L for i in range(M) for j in range(M) for k in range(M)]
    c = len(shifts)
    off = np.arange(c)[:, None]
    return dataclasses.replace(
        s, name="repeated", coor=np.concatenate([s.coor + d for d in shifts]), ptchg=np.tile(s.ptchg, c),
        epsgm6=np.tile(s.epsgm6, c), epsgm12=np.tile(s.epsgm12, c),
        exc1=np.concatenate([[0], (s.exc1[1:] + off * len(s.exc2)).ravel()]).astype(np.int32),
        exc2=(s.exc2 + off * n).ravel().astype(np.int32), poipt=(s.poipt + off * n).ravel().astype(np.int32),
        montype=np.tile(s.montype, c), box=tuple(M * L), nfft=tuple(M * g for g in s.nfft)), c


@pytest.fixture(scope="module")
def boxes():
    s = small_box()
    big, copies = repeated(s)
    assert big.nwaters >= 65536
    ref, eref = O.eforce(s, mode="parity")
    return s, big, copies, ref, eref


def joined(e):
    """Terms that do not depend on which pairs cross the box's faces."""
    return {"lj": e["e_vdw"] + e["e_vsym"], "el": e["e_el"] + e["e_lsym"], "corr": e["e_corr"], "self": e["e_self"],
            "rec": e["e_ew_receip"], "total": e["e_total"]}


@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
def test_gradient_and_energies(boxes, precision):
    s, big, copies, ref, eref = boxes
    fp64 = precision == MOIL_NB_FP64
    nb = Nonbonded(big, precision=precision)
    want = joined(eref)
    for _ in range(2):
        dpot, e = nb.eforce(big.coor)
        assert rel_rms(dpot.reshape(copies, -1), np.tile(ref.reshape(1, -1), (copies, 1))) <= (2.0 ** -25 if fp64 else 1e-5)
        got = joined(e)
        assert all(abs(got[k] / copies - want[k]) <= (1e-10 if fp64 else 1e-6) * energy_scale(eref) for k in want)
    nb.close()


@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
def test_derivatives_and_pressure(boxes, precision):
    s, big, copies, _, _ = boxes
    nb = Nonbonded(big, precision=precision)
    for got, want in zip(nb.adjoint(big.coor), O.adjoint(s)):
        assert rel_rms(got.reshape(copies, -1), np.tile(want, (copies, 1))) <= 1e-5
    mol, mass = S.molecules(s)
    want = O.pressure(s, mol, mass, mode="mi")[2]
    n = int(mol.max()) + 1
    nb.set_molecules(np.concatenate([mol + k * n for k in range(copies)]), np.tile(mass, copies))
    press = nb.pressure(big.coor, with_gradient=False)[2]
    nb.close()
    assert np.abs(press / copies - want).max() <= (1e-9 if precision == MOIL_NB_FP64 else 1e-5) * np.abs(want).sum()
