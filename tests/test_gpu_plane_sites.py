"""The PME planes' own selection of their sites, where it can go wrong: grids whose planes are too
small to queue all their sites at once, planes whose stencil wraps, the longest side, and more
sites than a block tests in one round.  Against the oracle, to the mixed path's tolerances."""
import ctypes

import numpy as np
import pytest

from conftest import rel_rms
from moil_fnrfd_gb300 import nb as NB
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("grid", [(4, 4, 4), (5, 4, 6), (4, 6, 128), (30, 32, 5)])
def test_small_and_long_planes(cfg0, grid, precision):
    s = cfg0.copy()
    s.nfft = grid
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, precision=precision)
    dpot, e = nb.eforce(s.coor)
    assert rel_rms(dpot, ref) <= (1e-5 if precision == MOIL_NB_MIXED else 2.0 ** -25)
    tol = 1e-5 if precision == MOIL_NB_MIXED else 1e-10
    assert abs(e["e_ew_receip"] - eref["e_ew_receip"]) <= tol * abs(eref["e_ew_receip"])
    nb.close()


@pytest.mark.parametrize("grid", [(10, 9, 8), (27, 50, 36), (96, 20, 6), (6, 75, 45), (40, 25, 24)])
def test_transform_lengths(cfg0, grid):
    """Lines of one, two and three passes along each axis, radices 2 to 10."""
    s = cfg0.copy()
    s.nfft = grid
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s)
    dpot, e = nb.eforce(s.coor)
    assert rel_rms(dpot, ref) <= 1e-5
    assert abs(e["e_ew_receip"] - eref["e_ew_receip"]) <= 1e-5 * abs(eref["e_ew_receip"])
    nb.close()


@pytest.mark.parametrize("natom", [1, 255, 16384, 16401, 33001])
def test_sites_past_one_round(natom):
    """The allocation-free sum on natom random charges (a block tests 16,384 sites per round)."""
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(natom))
    L, n = 40.0, natom
    x, q = rng.uniform(-L / 2, L / 2, size=(n, 3)), rng.normal(0.0, 0.5, size=n)
    s = S.MoilSystem(name="charges", coor=x, ptchg=q, epsgm6=np.zeros(n), epsgm12=np.zeros(n),
                     exc1=np.zeros(n + 1, np.int32), exc2=np.zeros(0, np.int32), spec1=np.zeros(0, np.int32),
                     spec2=np.zeros(0, np.int32), p14=np.zeros((0, 3)), poipt=np.arange(1, n + 1, dtype=np.int32),
                     montype=np.full(n, S.MON_ION, np.int32), box=(L, L, L), alpha=0.35, nfft=(40, 40, 40))
    ref, eref = O.pme(s, 0.35)
    fn = NB.load().moil_nb_pme_noalloc
    dc = torch.tensor(x, dtype=torch.float64, device="cuda")
    dq = torch.tensor(q, dtype=torch.float64, device="cuda")
    dd = torch.full_like(dc, float("nan"))
    torch.cuda.synchronize()
    e = ctypes.c_double()
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                   ctypes.POINTER(ctypes.c_int), ctypes.c_double, ctypes.c_double, ctypes.c_void_p,
                   ctypes.POINTER(ctypes.c_double), ctypes.c_void_p]
    rc = fn(dc.data_ptr(), dq.data_ptr(), n, (ctypes.c_double * 3)(L, L, L), (ctypes.c_int * 3)(40, 40, 40), 0.35, 1.0,
            dd.data_ptr(), ctypes.byref(e), None)
    assert rc == 0
    # a lone charge feels only its own images through the grid: its gradient is rounding
    got = dd.cpu().numpy()
    if n > 1:
        assert rel_rms(got, ref) <= 1e-5
    else:
        assert np.abs(got - ref).max() <= 1e-5 * abs(eref)
    assert abs(e.value - eref) <= 1e-5 * abs(eref)


@pytest.mark.parametrize("grid", [(10, 9, 8), (27, 50, 36), (96, 20, 6), (6, 75, 45), (5, 4, 125)])
def test_transform_lengths_fp64(cfg0, grid):
    """The plain path's passes: one, two and three along each axis, odd row counts."""
    s = cfg0.copy()
    s.nfft = grid
    ref, eref = O.eforce(s, mode="parity")
    nb = Nonbonded(s, precision=MOIL_NB_FP64)
    dpot, e = nb.eforce(s.coor)
    assert rel_rms(dpot, ref) <= 2.0 ** -25
    assert abs(e["e_ew_receip"] - eref["e_ew_receip"]) <= 1e-10 * abs(eref["e_ew_receip"])
    nb.close()
