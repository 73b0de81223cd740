"""The automatic water shape: half lists for large handles, whether a few of their atoms are ions or none, full
lists for small ones and for solutes in handles of up to 50,000 waters; the same in every replica
group (the gradient's bits do not depend on the grouping)."""
import numpy as np
import pytest

from conftest import ENERGY_TERMS, energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import WATER_FULL, WATER_HALF, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def ion_box(n_waters, n_ions, seed):
    """A water box with some of its molecules replaced by ions of alternating charge."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, box = n_waters + n_ions, ((n_waters + n_ions) / S.WATER_DENSITY) ** (1 / 3)
    sites = S._lattice_sites(int(np.ceil(n ** (1 / 3) - 1e-9)), box)
    oxy = sites[np.sort(rng.choice(len(sites), size=n, replace=False))] + rng.uniform(-0.3, 0.3, (n, 3))
    at = np.linspace(0, n - 1, n_ions).astype(int)
    b = S._Builder(arith=False)
    for k, x in enumerate(oxy[at]):
        b.add_monomer(x[None, :], [1.0 if k % 2 == 0 else -1.0], [0.0469], [S.rmin2_to_sigma(1.3638)], S.MON_ION)
    b.add_waters(S._place_waters(rng, np.delete(oxy, at, axis=0)))
    g = S.smooth_grid(box)
    return b.finish("ions", box, rvmx=9.0, relx=9.0, alpha=0.35, nfft=(g, g, g), seed=seed)


@pytest.mark.parametrize("name,want", [("ions_32000", WATER_HALF), ("ions_28000", WATER_FULL),
                                       ("waters_32000", WATER_HALF), ("solutes_35100", WATER_FULL),
                                       ("solutes_56160", WATER_HALF)])
def test_automatic_water_shape(name, want):
    if name.startswith("solutes"):
        s = S.config1()
    else:
        s = ion_box(2000, 2, 5) if name.startswith("ions") else S.water_box(2000, 39.12, 6)
    n = int(name.split("_")[1])
    batch = [s] * (n // s.nwaters)
    ref, eref = O.eforce(s, mode="parity")
    bits = []
    for groups in (1, 2):
        nb = Nonbonded(batch, groups=groups)
        assert nb.groups() == groups and nb.shape()["water_kernel"] == want
        dps, es = nb.eforce()
        nb.close()
        assert rel_rms(dps[-1], ref) <= 1e-5
        assert all(abs(es[-1][k] - eref[k]) <= 1e-6 * energy_scale(eref) for k in ENERGY_TERMS + ("e_total",))
        bits.append(np.concatenate(dps))
    assert np.array_equal(bits[0], bits[1])
