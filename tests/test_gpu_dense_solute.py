"""Waters inside a dense solute, whose lists of non-water atoms pass 64 entries for every lane that
shares them (at 8 and 4 lanes per water), so the lanes flush their partial gradients into the row's shared
sums while they run through that list.  Against the oracle in parity mode: 1e-5 of the gradient and
1e-6 of the energy-term scale per term."""
import numpy as np
import pytest

from conftest import ENERGY_TERMS, energy_scale, rel_rms
from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import WATER_FULL, Nonbonded
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BOX, RADIUS = 30.0, 12.2


def waters_in_a_dense_solute(seed=5):
    """Single-atom monomers of alternating charge on a 1.9 Å lattice inside a sphere of 12.2 Å, three waters in
    holes around its centre and a shell of waters outside."""
    rng = np.random.Generator(np.random.PCG64(seed))
    g = 1.9 * np.arange(-7, 8)
    grid = np.stack([v.ravel() for v in np.meshgrid(g, g, g, indexing="ij")], axis=1)
    parity = np.rint(grid / 1.9).astype(int).sum(1) % 2
    holes = np.array([[0.0, 0.0, 0.0], [0.0, 3.8, 3.8], [-3.8, 0.0, -3.8]])
    ok = (grid ** 2).sum(1) <= RADIUS ** 2
    ok &= (((grid[:, None] - holes[None]) ** 2).sum(2) > 2.4 ** 2).all(1)
    xyz, sign = grid[ok] + rng.uniform(-0.05, 0.05, (int(ok.sum()), 3)), np.where(parity[ok] == 1, 1.0, -1.0)
    q = 0.3 * sign
    q -= q.mean()
    b = S._Builder(arith=True)
    for x, c in zip(xyz, q):
        b.add_monomer(x[None, :], [c], [0.05], [1.6], S.MON_OTHER)
    sites = S._lattice_sites(10, BOX) + rng.uniform(-0.2, 0.2, (1000, 3))
    sites = sites[(sites ** 2).sum(1) > (RADIUS + 2.4) ** 2]
    b.add_waters(S._place_waters(rng, np.concatenate([holes, sites])))
    s = b.finish("dense_solute", BOX, rvmx=9.0, relx=9.0, alpha=0.35, nfft=(30, 30, 30), seed=seed)
    return s, xyz, holes


@pytest.mark.parametrize("filler", [3, 11], ids=["8_lanes", "4_lanes"])
def test_long_atom_lists_match_oracle(filler):
    s, xyz, holes = waters_in_a_dense_solute()
    # list entries of a water: atoms within cutoff + skin + 1.1 Å of its oxygen
    near = (((holes[:, None] - xyz[None]) ** 2).sum(2) <= 11.1 ** 2).sum(1)
    assert (near > 8 * 64).all()
    box = S.water_box(3203, (3203 / S.WATER_DENSITY) ** (1 / 3), 10)
    nb = Nonbonded([s] + [box] * filler, shape=dict(water_kernel=WATER_FULL), groups=1)
    ref, eref = O.eforce(s, mode="parity")
    scale = energy_scale(eref)
    for _ in range(2):
        dps, es = nb.eforce()
        assert rel_rms(dps[0], ref) <= 1e-5
        w = 3 * (s.nwaters - len(holes))
        assert rel_rms(dps[0][-w - 9:-w], ref[-w - 9:-w]) <= 1e-5          # the waters in the holes
        assert all(abs(es[0][k] - eref[k]) <= 1e-6 * scale for k in ENERGY_TERMS + ("e_total",))
    nb.close()


def test_group_without_atoms_gives_the_same_bits():
    """Water boxes in a replica group of their own beside a group with the solute: the kernels are chosen by what
    the whole handle holds."""
    s = waters_in_a_dense_solute()[0]
    box = S.water_box(800, (800 / S.WATER_DENSITY) ** (1 / 3), 10)
    out = []
    for groups in (1, 2):
        nb = Nonbonded([s, box], groups=groups)
        assert nb.groups() == groups
        dps, es = nb.eforce()
        out.append((np.concatenate(dps), [e["e_total"] for e in es]))
        nb.close()
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
