"""The reciprocal sum of the allocation-free entry point takes any coordinate without leaving its grid: absurd ones
(10^8 to 10^30 Å, NaN, infinities) give a finite gradient for the other atoms' kernels to add up, and the
next call on sane ones is right."""
import numpy as np
import pytest

from conftest import rel_rms
from moil_fnrfd_gb300 import systems as S
from oracle import oracle as O
from test_zz_no_alloc import noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(4, 4, 4), (20, 20, 20), (64, 64, 64)])
def test_absurd_coordinates_stay_on_the_grid(grid):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(2))
    s = S.config0()
    s.nfft = grid
    x = s.coor.copy()
    x[:300] = rng.choice([-1.0, 1.0], (300, 3)) * 10.0 ** rng.uniform(8.0, 30.0, (300, 3))
    x[300:330] = rng.choice([np.nan, np.inf, -np.inf], (30, 3))
    far = s.copy()
    far.coor = x
    dpot, e = noalloc(torch, far)
    assert np.isfinite(dpot).all() and np.isfinite(e)
    ref, e_ref = O.pme(s, s.alpha)
    dpot, e = noalloc(torch, s)
    assert rel_rms(dpot, ref) <= 1e-5 and abs(e - e_ref) <= 1e-6 * abs(e_ref)
